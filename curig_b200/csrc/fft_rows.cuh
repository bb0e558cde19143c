// Row transforms of the oversampled planes, hand-written (Stockham, radices 2
// to 16, a row or pair of rows per group of threads, exchanges through shared
// memory), one kernel per row length and precision.
//
// The reference transforms every plane with a batched 2-D cuFFT
// (cuft.cu:127-143).  Only the image's columns (and rows) of a transformed
// plane are used, so the 2-D transform is two passes of rows here, and what
// surrounds them is part of the pass that touches the data:
//   X_M2D  grid row -> transform -> its image columns, transposed into T
//   Y_M2D  row of T -> transform -> its image rows, in place
//   Y_D2M  image rows of a row of T (zeros elsewhere) -> transform -> the row
//   X_D2M  image columns gathered from T (zeros elsewhere) -> transform -> grid row
// T is [z][x'][y], x' over the image columns (kernels.cu).  With G = the
// grid's bytes and half of the columns and rows in the image, a direction moves
// 1.5 G + 0.75 G where library rows, separate transposes, zero padding and
// full rows moved 4 G and more.  The grid's side is limited to the window of
// cells that the points reach (FftGeom): rows outside it are not transformed,
// cells outside it are taken as zero and not written (uv coverage to 0.3
// cycles per pixel leaves 0.4 of the cells).
//
// Elements: 16 bytes.  FP64 one complex number; FP32 the same element of two
// rows, real parts and imaginary parts packed, so that the packed FP32
// instructions (add / mul / fma .f32x2) do both rows in one issue slot and a
// shared-memory access moves both (one row per thread group was bound by
// instruction issue: 2048^2 image, 18 planes, x rows 1.27 ms).
//
// Threads: T threads hold a unit (at most 18 elements each: one radix-16, two
// radix-8, ... butterflies a stage), reads of the first stage come from global
// memory and writes of the last go there, so a unit of s stages makes s - 1
// trips through shared memory.  F = 2 units interleave lane by lane where they
// fit, so a warp's transposed accesses are 32-byte sectors.
//
// The length is a template parameter: radices, strides and butterfly counts are
// constants, shared-memory accesses take immediate offsets and a kernel holds
// only its own radices.  (One kernel that switched over the radices at run time
// executed 29 instructions per element and stage and stalled on instruction
// fetches: FP64 4096-point x rows, 98304 of them, 2.78 ms.)  The two directions
// share a kernel: only the first stage's loads and the last one's stores
// differ, and the forward direction is the inverse one with real and imaginary
// parts swapped on both sides.
#pragma once

#include "fft.h"
#include "plan.h"

namespace curig {

template <typename T> using C = typename cplx_t<T>::type;

// ------------------------------------------------------------------ arithmetic
// V2: two FP32 values in one 64-bit register pair (packed instructions).
struct V2 {
    unsigned long long v;
};
__device__ __forceinline__ V2 pack2(float a, float b) {
    V2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(V2 a, float &x, float &y) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
}
__device__ __forceinline__ V2 add(V2 a, V2 b) {
    V2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ V2 mul(V2 a, V2 b) {
    V2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ V2 madd(V2 a, V2 b, V2 c) {
    V2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ V2 neg(V2 a) { return V2{a.v ^ 0x8000000080000000ULL}; }
__device__ __forceinline__ V2 sub(V2 a, V2 b) { return madd(b, pack2(-1.f, -1.f), a); }

__device__ __forceinline__ double add(double a, double b) { return a + b; }
__device__ __forceinline__ double sub(double a, double b) { return a - b; }
__device__ __forceinline__ double mul(double a, double b) { return a * b; }
__device__ __forceinline__ double madd(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ double neg(double a) { return -a; }

template <typename S> struct Lit;                      // a constant in every lane of S
template <> struct Lit<V2> {
    static __device__ __forceinline__ V2 of(double c) { return pack2((float)c, (float)c); }
};
template <> struct Lit<double> {
    static __device__ __forceinline__ double of(double c) { return c; }
};

template <typename S> struct __align__(16) Cx {
    S x, y;
};
// twiddle: e^{i a} with the negated imaginary part at hand (no negated
// operands in the packed instructions)
template <typename S> struct Tw {
    S x, y, ny;
};
template <typename S> __device__ __forceinline__ Cx<S> cadd(Cx<S> a, Cx<S> b) { return {add(a.x, b.x), add(a.y, b.y)}; }
template <typename S> __device__ __forceinline__ Cx<S> csub(Cx<S> a, Cx<S> b) { return {sub(a.x, b.x), sub(a.y, b.y)}; }
template <typename S> __device__ __forceinline__ Cx<S> cmul(Cx<S> a, Tw<S> w) {
    return {madd(a.y, w.ny, mul(a.x, w.x)), madd(a.y, w.x, mul(a.x, w.y))};
}
template <typename S> __device__ __forceinline__ Tw<S> tmul(Tw<S> a, Tw<S> b) {
    const S y = madd(a.y, b.x, mul(a.x, b.y));
    return {madd(a.y, b.ny, mul(a.x, b.x)), y, neg(y)};
}

// ------------------------------------------------------------------ small transforms
// cos / sin of 2 pi a / n at compile time: octant reduction, Taylor series.
constexpr double taylor_cos(double x) {
    double t = 1.0, s = 1.0;
    for (int k = 1; k < 14; ++k) {
        t *= -x * x / ((2.0 * k - 1.0) * (2.0 * k));
        s += t;
    }
    return s;
}
constexpr double taylor_sin(double x) {
    double t = x, s = x;
    for (int k = 1; k < 14; ++k) {
        t *= -x * x / ((2.0 * k) * (2.0 * k + 1.0));
        s += t;
    }
    return s;
}
struct CosSin {
    double c, s;
};
constexpr CosSin unit_root(int a, int n) {
    a %= n;
    double sg = 1.0, cg = 1.0;
    if (2 * a > n) { a = n - a; sg = -1.0; }           // angle pi b / n, b = 2 a in [0, n]
    int b = 2 * a;
    if (2 * b > n) { b = n - b; cg = -1.0; }           // angle in [0, pi / 2]
    const int c = 2 * b;                               // (pi / 2) c / n, c in [0, n]
    const double h = PI_D / 2.0;
    if (2 * c > n) return CosSin{cg * taylor_sin(h * (n - c) / n), sg * taylor_cos(h * (n - c) / n)};
    return CosSin{cg * taylor_cos(h * c / n), sg * taylor_sin(h * c / n)};
}
constexpr int gcd_int(int a, int b) { return b == 0 ? a : gcd_int(b, a % b); }

template <int I> struct ic {
    static constexpr int v = I;
};
template <int N, int I = 0, class Fn> __device__ __forceinline__ void static_for(Fn &&f) {
    if constexpr (I < N) {
        f(ic<I>{});
        static_for<N, I + 1>(f);
    }
}

// a times e^{2 pi i A / N}
template <int A, int N, typename S> __device__ __forceinline__ Cx<S> cmul_root(Cx<S> a) {
    constexpr int r = A % N;
    if constexpr (r == 0) return a;
    else if constexpr (4 * r == N) return {neg(a.y), a.x};
    else if constexpr (2 * r == N) return {neg(a.x), neg(a.y)};
    else if constexpr (4 * r == 3 * N) return {a.y, neg(a.x)};
    else {
        constexpr CosSin w = unit_root(r, N);
        const S c = Lit<S>::of(w.c), s = Lit<S>::of(w.s), ns = Lit<S>::of(-w.s);
        return {madd(a.y, ns, mul(a.x, c)), madd(a.y, c, mul(a.x, s))};
    }
}

// R-point transforms, e^{+2 pi i n k / R}
template <int R> struct Dft;

template <> struct Dft<2> {
    template <typename S> static __device__ __forceinline__ void run(Cx<S> (&v)[2]) {
        const Cx<S> a = v[0], b = v[1];
        v[0] = cadd(a, b);
        v[1] = csub(a, b);
    }
};
template <> struct Dft<3> {
    template <typename S> static __device__ __forceinline__ void run(Cx<S> (&v)[3]) {
        constexpr CosSin w = unit_root(1, 3);
        const S s = Lit<S>::of(w.s), ns = Lit<S>::of(-w.s), h = Lit<S>::of(-0.5);
        const Cx<S> t = cadd(v[1], v[2]), d = csub(v[1], v[2]);
        const Cx<S> m = {madd(t.x, h, v[0].x), madd(t.y, h, v[0].y)};
        v[0] = cadd(v[0], t);
        v[1] = {madd(d.y, ns, m.x), madd(d.x, s, m.y)};
        v[2] = {madd(d.y, s, m.x), madd(d.x, ns, m.y)};
    }
};
template <> struct Dft<4> {
    template <typename S> static __device__ __forceinline__ void run(Cx<S> (&v)[4]) {
        const Cx<S> a = cadd(v[0], v[2]), b = csub(v[0], v[2]), c = cadd(v[1], v[3]);
        const Cx<S> d = csub(v[1], v[3]);
        v[0] = cadd(a, c);
        v[2] = csub(a, c);
        v[1] = {sub(b.x, d.y), add(b.y, d.x)};
        v[3] = {add(b.x, d.y), sub(b.y, d.x)};
    }
};
template <> struct Dft<5> {
    template <typename S> static __device__ __forceinline__ void run(Cx<S> (&v)[5]) {
        constexpr CosSin w1 = unit_root(1, 5), w2 = unit_root(2, 5);
        const S c1 = Lit<S>::of(w1.c), c2 = Lit<S>::of(w2.c);
        const S s1 = Lit<S>::of(w1.s), s2 = Lit<S>::of(w2.s), n1 = Lit<S>::of(-w1.s);
        const Cx<S> a = cadd(v[1], v[4]), b = csub(v[1], v[4]), c = cadd(v[2], v[3]), d = csub(v[2], v[3]);
        const Cx<S> m1 = {madd(c.x, c2, madd(a.x, c1, v[0].x)), madd(c.y, c2, madd(a.y, c1, v[0].y))};
        const Cx<S> m2 = {madd(c.x, c1, madd(a.x, c2, v[0].x)), madd(c.y, c1, madd(a.y, c2, v[0].y))};
        const Cx<S> e1 = {madd(d.x, s2, mul(b.x, s1)), madd(d.y, s2, mul(b.y, s1))};
        const Cx<S> e2 = {madd(d.x, n1, mul(b.x, s2)), madd(d.y, n1, mul(b.y, s2))};
        v[0] = cadd(v[0], cadd(a, c));
        v[1] = {sub(m1.x, e1.y), add(m1.y, e1.x)};
        v[4] = {add(m1.x, e1.y), sub(m1.y, e1.x)};
        v[2] = {sub(m2.x, e2.y), add(m2.y, e2.x)};
        v[3] = {add(m2.x, e2.y), sub(m2.y, e2.x)};
    }
};

// index k with k mod R1 = k1, k mod R2 = k2 (coprime R1, R2)
constexpr int crt_index(int R1, int R2, int k1, int k2) {
    for (int k = 0; k < R1 * R2; ++k)
        if (k % R1 == k1 && k % R2 == k2) return k;
    return -1;
}

// R = R1 R2: prime-factor maps for coprime factors (no twiddles), else
// Cooley-Tukey with compile-time twiddles.
template <int R1, int R2, typename S> __device__ __forceinline__ void dft_product(Cx<S> (&v)[R1 * R2]) {
    using Z = Cx<S>;
    constexpr int R = R1 * R2;
    constexpr bool pfa = gcd_int(R1, R2) == 1;
    Z u[R1][R2];
    static_for<R2>([&](auto n2) {
        Z a[R1];
        static_for<R1>([&](auto n1) {
            a[n1.v] = v[pfa ? (R2 * n1.v + R1 * n2.v) % R : R2 * n1.v + n2.v];
        });
        Dft<R1>::run(a);
        static_for<R1>([&](auto k1) {
            u[k1.v][n2.v] = pfa ? a[k1.v] : cmul_root<decltype(n2)::v * decltype(k1)::v, R>(a[k1.v]);
        });
    });
    static_for<R1>([&](auto k1) {
        Dft<R2>::run(u[k1.v]);
        static_for<R2>([&](auto k2) {
            constexpr int o = pfa ? crt_index(R1, R2, decltype(k1)::v, decltype(k2)::v)
                                  : decltype(k1)::v + R1 * decltype(k2)::v;
            v[o] = u[k1.v][k2.v];
        });
    });
}
#define CURIG_DFT(R, R1, R2)                                                                       \
    template <> struct Dft<R> {                                                                    \
        template <typename S> static __device__ __forceinline__ void run(Cx<S> (&v)[R]) {          \
            dft_product<R1, R2>(v);                                                                \
        }                                                                                          \
    };
CURIG_DFT(6, 2, 3)
CURIG_DFT(8, 2, 4)
CURIG_DFT(9, 3, 3)
CURIG_DFT(10, 2, 5)
CURIG_DFT(12, 3, 4)
CURIG_DFT(15, 3, 5)
CURIG_DFT(16, 4, 4)
#undef CURIG_DFT

// ------------------------------------------------------------------ lengths
// Radices and thread layout of one row length.  Position i of a unit in
// shared memory: R0 elements, then `pad` unused ones.  R0 + pad is odd, so the
// strided writes of the first stage spread over the banks, and every later
// stride is a multiple of R0, so positions advance by one constant per element.
// SP = 2: the unit is half of a row of 2 N elements, its even or its odd outputs
// (X[2 k + c] is the N-point transform of (x[i] + (-1)^c x[i + N]) w^(c i), w the
// 2N-th root): rows longer than one unit takes two CTAs, which read the row
// twice (from L2 the second time) and need nothing of each other.
template <bool X, int SP_, int N_, int T_, int FX, int GX, int GY, int R0, int R1, int R2, int R3, int R4>
struct FftLen {
    static constexpr bool x = X;
    static constexpr int SP = SP_;
    using Half = FftLen<X, 2, N_, T_, FX, GX, GY, R0, R1, R2, R3, R4>;
    static constexpr int N = N_, T = T_, F = X && SP == 1 ? FX : 1, G = SP > 1 ? 1 : X ? GX : GY;
    static constexpr int R[5] = {R0, R1, R2, R3, R4};
    static constexpr int stages = R2 == 1 ? 2 : R3 == 1 ? 3 : R4 == 1 ? 4 : 5;
    static constexpr int pad = R0 % 2 == 0 ? 1 : 0;
    static constexpr int pitch = N + pad * (N / R0);
    static constexpr int threads = (T * F * G + 31) / 32 * 32;
    static constexpr size_t smem = (size_t)pitch * F * G * 16;
    static constexpr int Ns(int s) { return s == 0 ? 1 : s == 1 ? R0 : s == 2 ? R0 * R1 : s == 3 ? R0 * R1 * R2 : R0 * R1 * R2 * R3; }
    static constexpr int radix(int s) { return s == 0 ? R0 : s == 1 ? R1 : s == 2 ? R2 : s == 3 ? R3 : R4; }
    static constexpr int powers(int r) { return r > 8 ? 4 : r > 4 ? 3 : r > 2 ? 2 : 1; }      // 1, 2, 4, 8 below r
    // offset of stage s's twiddle table [powers][Ns]
    static constexpr int tw(int s) { return s <= 1 ? 0 : tw(s - 1) + powers(radix(s - 1)) * Ns(s - 1); }
    static constexpr int tw_split() { return tw(stages - 1) + powers(radix(stages - 1)) * Ns(stages - 1); }   // w^j, j < N / R0
    __device__ static __forceinline__ int pos(int i) { return pad ? i + i / R0 : i; }
    static_assert(R0 * R1 * R2 * R3 * R4 == N && threads <= 512 && smem <= 72 * 1024, "row length");
};

template <typename T> struct lane_t;
template <> struct lane_t<float> { using type = V2; };
template <> struct lane_t<double> { using type = double; };

// ------------------------------------------------------------------ passes
// Twiddles w^q, w = e^{2 pi i k / (Ns R)} of one butterfly: powers 1, 2, 4 and
// 8 from the table (tb, a column of it), the others products of those.
template <typename S> __device__ __forceinline__ Tw<S> tw_get(const Cx<S> *__restrict__ tb) {
    const Cx<S> w = *tb;
    return Tw<S>{w.x, w.y, neg(w.y)};
}
template <int R, int Ns, typename S>
__device__ __forceinline__ void twiddle(Cx<S> (&v)[R], const Cx<S> *__restrict__ tb) {
    Tw<S> w[8];
    static_for<8>([&](auto q) {
        constexpr int Q = decltype(q)::v, H = Q >= 4 ? 4 : Q >= 2 ? 2 : 1;
        if constexpr (Q > 0 && Q < R) {
            if constexpr (Q == H) w[Q] = tw_get(tb + (Q == 1 ? 0 : Q == 2 ? 1 : 2) * Ns);
            else w[Q] = tmul(w[H], w[Q - H]);
            v[Q] = cmul(v[Q], w[Q]);
        }
    });
    if constexpr (R > 8) {
        const Tw<S> w8 = tw_get(tb + 3 * Ns);
        v[8] = cmul(v[8], w8);
        static_for<8>([&](auto q) {
            constexpr int Q = decltype(q)::v;
            if constexpr (Q > 0 && Q + 8 < R) v[Q + 8] = cmul(v[Q + 8], tmul(w8, w[Q]));
        });
    }
}

// Row data passes through once: loads that leave L1 to the twiddle tables, and
// give 0 without reading where `on` is false (predicated, so that the loads of
// a butterfly issue back to back).
__device__ __forceinline__ float2 ld_once(const float2 *p, bool on) {
    float2 v;
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %3, 0;\n\tmov.f32 %0, 0f00000000;\n\tmov.f32 %1, 0f00000000;\n\t"
                 "@p ld.global.L1::no_allocate.v2.f32 {%0, %1}, [%2];\n\t}"
                 : "=&f"(v.x), "=&f"(v.y) : "l"(p), "r"((int)on));
    return v;
}
__device__ __forceinline__ float4 ld_once(const float4 *p, bool on) {
    float4 v;
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\tmov.f32 %0, 0f00000000;\n\tmov.f32 %1, 0f00000000;\n\t"
                 "mov.f32 %2, 0f00000000;\n\tmov.f32 %3, 0f00000000;\n\t"
                 "@p ld.global.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}"
                 : "=&f"(v.x), "=&f"(v.y), "=&f"(v.z), "=&f"(v.w) : "l"(p), "r"((int)on));
    return v;
}
__device__ __forceinline__ double2 ld_once(const double2 *p, bool on) {
    double2 v;
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %3, 0;\n\tmov.f64 %0, 0d0000000000000000;\n\t"
                 "mov.f64 %1, 0d0000000000000000;\n\t"
                 "@p ld.global.L1::no_allocate.v2.f64 {%0, %1}, [%2];\n\t}"
                 : "=&d"(v.x), "=&d"(v.y) : "l"(p), "r"((int)on));
    return v;
}

// The buffers that a launch reads and writes, for the index checks of the
// bounds-checked build: n elements at p, aligned to their size, inside the
// buffer.  Nothing of it is left in the regular build, whose kernels are the same
// with and without; an unused flag pointer in FftGeom was enough to change their
// registers (1000^2 image, FP64, ms2dirty's passes 351 -> 355 us), so that one has none.
#ifdef CURIG_BOUNDS_CHECK
#define ROW_FLAGS(g) (g).dbg
#else
#define ROW_FLAGS(g) nullptr
#endif
template <typename T> struct Limits {
    const C<T> *in0, *in1, *out0, *out1;
    int *flags;
    __device__ __forceinline__ static bool inside(const C<T> *p, int n, const C<T> *a, const C<T> *b) {
        return p >= a && p + n <= b && (size_t)p % (n * sizeof(C<T>)) == 0;
    }
    __device__ __forceinline__ bool reads(const C<T> *p, int n) const { return inside(p, n, in0, in1); }
    __device__ __forceinline__ bool writes(const C<T> *p, int n) const { return inside(p, n, out0, out1); }
};

// Where a unit comes from and goes to: element i of its row (FP64) or of its
// two rows (FP32; the second `row2` elements after the first, absent where two
// is false).  In T the X passes' two rows are neighbours (y, y + 1).
template <typename T, bool X, int SP> struct RowMem {
    using S = typename lane_t<T>::type;
    static constexpr bool in_place = !X && SP == 2;
    const C<T> *in;
    C<T> *out;
    long long row2;
    bool two, act, m2d, odd;       // odd: SP = 2, the odd outputs
    int lo, hi, m;                 // elements outside the image: [lo, hi); row length of T
    int w0, w1;                    // elements of the grid side inside the window
    Limits<T> lim;
    __device__ __forceinline__ Cx<S> row(int i, bool on) const {
        on = on && IN_BOUNDS(lim.reads(in + i, 1) && lim.reads(in + i + row2, 1), lim.flags);
        if constexpr (sizeof(T) == 8) {
            const C<T> u = ld_once(in + i, on);
            return Cx<S>{u.x, u.y};
        } else {
            const C<T> u = ld_once(in + i, on), w = ld_once(in + i + row2, on);
            return Cx<S>{pack2(u.x, w.x), pack2(u.y, w.y)};
        }
    }
    __device__ __forceinline__ Cx<S> col(int i, bool on) const {
        const C<T> *a = in + (long long)(i < lo ? i : i - hi + lo) * m;
        on = on && IN_BOUNDS(lim.reads(a, 16 / (int)sizeof(C<T>)), lim.flags);
        if constexpr (sizeof(T) == 8) {
            const C<T> u = ld_once(a, on);
            return Cx<S>{u.x, u.y};
        } else {
            const float4 u = ld_once(reinterpret_cast<const float4 *>(a), on);
            return Cx<S>{pack2(u.x, u.z), pack2(u.y, u.w)};
        }
    }
    __device__ __forceinline__ void put_row(int i, Cx<S> v) const {
        if (!IN_BOUNDS(lim.writes(out + i, 1) && lim.writes(out + i + row2, 1), lim.flags)) return;
        if constexpr (sizeof(T) == 8) out[i] = C<T>{v.x, v.y};
        else {
            float4 u;
            unpack2(v.x, u.x, u.z);
            unpack2(v.y, u.y, u.w);
            out[i] = C<T>{u.x, u.y};
            if (two) out[i + row2] = C<T>{u.z, u.w};
        }
    }
    __device__ __forceinline__ void put_col(int i, Cx<S> v) const {
        C<T> *o = out + (long long)(i < lo ? i : i - hi + lo) * m;
        if (!IN_BOUNDS(lim.writes(o, 16 / (int)sizeof(C<T>)), lim.flags)) return;
        if constexpr (sizeof(T) == 8) *o = C<T>{v.x, v.y};
        else {
            float4 u;
            unpack2(v.x, u.x, u.z);
            unpack2(v.y, u.y, u.w);
            *reinterpret_cast<float4 *>(o) = u;
        }
    }
    __device__ __forceinline__ static Cx<S> swap(Cx<S> v) { return Cx<S>{v.y, v.x}; }
    // elements j + q STEP, q < R, as the transform takes them (the direction is
    // uniform over the launch; the forward one swaps real and imaginary parts);
    // M2D and the part of the row, i + base, fixed at compile time
    template <bool M2D> __device__ __forceinline__ Cx<S> elem(int i) const {
        if constexpr (M2D) return row(i, i >= w0 && i < w1);
        else {
            const bool on = i < lo || i >= hi;
            return swap(X ? col(i, on) : row(i, on));
        }
    }
    template <bool M2D, int R, int STEP>
    __device__ __forceinline__ void load_dir(int j, Cx<S> (&v)[R], const Cx<S> *__restrict__ tw) const {
        if constexpr (SP == 1) {
#pragma unroll
            for (int q = 0; q < R; ++q) v[q] = elem<M2D>(j + q * STEP);
        } else if (odd) {
            const Tw<S> wj = tw_get(tw);
            static_for<R>([&](auto q) {
                constexpr int Q = decltype(q)::v;
                const Cx<S> a = elem<M2D>(j + Q * STEP), b = elem<M2D>(j + (Q + R) * STEP);
                v[Q] = cmul(cmul_root<Q, 2 * R>(csub(a, b)), wj);
            });
        } else {
#pragma unroll
            for (int q = 0; q < R; ++q) v[q] = cadd(elem<M2D>(j + q * STEP), elem<M2D>(j + (q + R) * STEP));
        }
    }
    template <int R, int STEP> __device__ __forceinline__ void load(int j, Cx<S> (&v)[R], const Cx<S> *__restrict__ tw) const {
        if (m2d) load_dir<true, R, STEP>(j, v, tw);
        else load_dir<false, R, STEP>(j, v, tw);
    }
    template <int R, int STEP> __device__ __forceinline__ void store(int j, const Cx<S> (&v)[R]) const {
        const int c = SP == 2 && odd ? 1 : 0;
        if (m2d) {
#pragma unroll
            for (int q = 0; q < R; ++q) {
                const int i = SP * (j + q * STEP) + c;
                if (i < lo || i >= hi) {
                    if (X) put_col(i, v[q]);
                    else put_row(i, v[q]);
                }
            }
        } else {
#pragma unroll
            for (int q = 0; q < R; ++q) {
                const int i = SP * (j + q * STEP) + c;
                if (i >= w0 && i < w1) put_row(i, swap(v[q]));
            }
        }
    }
};

// Stage K of length L: butterflies j = t, t + T, ...; reads from global memory
// (first stage) or from the unit's shared buffer, twiddles, R-point transform,
// writes to the buffer in the order of the next stage or (last stage) to
// global memory.  Reads of the buffer are complete in every thread before it
// is overwritten.  Idle threads repeat the last butterfly and write nothing
// (conditional loads would put v into local memory).
template <class L, int K, typename S, class Mem>
__device__ __forceinline__ void fft_stage(int t, const Cx<S> *__restrict__ tw, Cx<S> *sm, const Mem &mem) {
    constexpr int R = L::radix(K), Ns = L::Ns(K), nbf = L::N / R, NB = (nbf + L::T - 1) / L::T;
    constexpr bool last = K == L::stages - 1, ragged = NB * L::T > nbf || L::T * L::F * L::G % 32 != 0;
    Cx<S> v[NB][R];
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        const int j = ragged ? min(t + b * L::T, nbf - 1) : t + b * L::T;
        if constexpr (K == 0) {
            mem.template load<R, nbf>(j, v[b], tw + L::tw_split() + j);
        } else {
            constexpr int step = (nbf + L::pad * (nbf / L::R[0])) * L::F;
            const Cx<S> *r = sm + L::pos(j) * L::F;
#pragma unroll
            for (int q = 0; q < R; ++q) v[b][q] = r[q * step];
            twiddle<R, Ns>(v[b], tw + L::tw(K) + j % Ns);
        }
        Dft<R>::run(v[b]);
    }
    if (K > 0 && !last) __syncthreads();
    // the halves of a row transformed in place: both have read it before either writes
    if constexpr (K == 0 && Mem::in_place) {
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        const int j = t + b * L::T;
        if (ragged && j >= nbf) continue;
        if constexpr (last) {
            if (mem.act) mem.template store<R, Ns>(j, v[b]);
        } else {
            constexpr int step = (K == 0 ? 1 : Ns + L::pad * (Ns / L::R[0])) * L::F;
            Cx<S> *w = sm + (K == 0 ? j * (R + L::pad) : L::pos(j + j / Ns * (Ns * (R - 1)))) * L::F;
#pragma unroll
            for (int q = 0; q < R; ++q) w[q * step] = v[b][q];
        }
    }
    if constexpr (!last) __syncthreads();
}

// Bound by the latency of its global loads at the 16 warps an SM that 128 registers
// leave: at 8192 points in two halves (one FP32 plane, ncu) issue slots are 31 to
// 38 % busy, DRAM 28 to 33 %, L1 45 to 72 %, and waiting for a load is the
// longest stall.  The X passes access T in 16 bytes of a 32-byte sector (F = 1),
// and the halves' interleaved outputs do the same on the grid.
//
// The units of one CTA: tid = (g T + t) F + f; unit g F + f of the CTA, F units
// interleaved element by element in shared memory.
template <typename T, class L>
__global__ void __launch_bounds__(L::threads, 512 / L::threads)
k_fft_rows(int m2d, FftGeom g, const Cx<typename lane_t<T>::type> *__restrict__ tw, const C<T> *src, C<T> *dst,
           long long rows) {
    using S = typename lane_t<T>::type;
    constexpr int PER = sizeof(T) == 4 ? 2 : 1;        // rows of a unit
    extern __shared__ __align__(16) unsigned char smem[];
    const int f = threadIdx.x % L::F, u = threadIdx.x / L::F;
    const int grp = min(u / L::T, L::G - 1), t = u - grp * L::T;
    Cx<S> *sm = reinterpret_cast<Cx<S> *>(smem) + grp * L::pitch * L::F + f;
    const long long want = (((long long)(blockIdx.x / L::SP) * L::G + grp) * L::F + f) * PER;
    RowMem<T, L::x, L::SP> mem;
    const long long ncell = (long long)g.nf3 * g.nf2 * g.nf1, nt = (long long)g.nf3 * g.ny * g.nf2;
    mem.lim = Limits<T>{src, src + (L::x && m2d ? ncell : nt), dst, dst + (L::x && !m2d ? ncell : nt), ROW_FLAGS(g)};
    mem.act = t < L::T && want < rows;                 // (idle threads read a unit again and write nothing)
    const long long row = want < rows ? want : 0;
    mem.m2d = m2d != 0;
    mem.two = row + 1 < rows;
    // X passes: row = z (y1 - y0) + y - y0; Y passes: row = z ny + x'
    if constexpr (L::x) {
        const long long z = row / (g.y1 - g.y0), y = g.y0 + (row - z * (g.y1 - g.y0));
        const long long tr = z * g.ny * (long long)g.nf2 + y, gr = (z * g.nf2 + y) * g.nf1;
        mem.in = src + (m2d ? gr : tr);
        mem.out = dst + (m2d ? tr : gr);
        mem.lo = g.ny - g.ny / 2;
        mem.hi = g.nf1 - g.ny / 2;
        mem.w0 = g.x0;
        mem.w1 = g.x1;
    } else {
        mem.in = src + row * g.nf2;
        mem.out = dst + row * g.nf2;
        mem.lo = g.nx - g.nx / 2;
        mem.hi = g.nf2 - g.nx / 2;
        mem.w0 = g.y0;
        mem.w1 = g.y1;
    }
    mem.odd = L::SP == 2 && blockIdx.x % 2 == 1;
    mem.row2 = mem.two ? L::SP * L::N : 0;
    mem.m = g.nf2;
    static_for<L::stages>([&](auto k) { fft_stage<L, decltype(k)::v>(t, tw, sm, mem); });
}

// ------------------------------------------------------------------ third axis (generic 3-D NUFFT)
// The planes' series along z at the integer modes k3 and the corrections, one
// line (x', y) of T a unit: m2d reads T[z][x'][y], transforms along z, writes
// fk[ix][iy][k3 + n3/2] divided by psi1 psi2 psi3; d2m the adjoint.  In FP64
// throughout, as the direct series (k_correct3_*) that other lengths keep; that
// one took n3 or nf3 terms per value with strided reads: 128^3 modes, 256
// planes, FP32 storage, 2165 us (d2m) and 604 us (m2d).
template <typename T> struct ZMem {
    const C<T> *in;
    C<T> *out;
    long long plane;
    int n3, nf3;
    const double *psi3;
    double den;
    bool m2d, act;
    Limits<T> lim;
    // mode index of grid index i, or -1
    __device__ __forceinline__ int mode(int i) const {
        return i < n3 - n3 / 2 ? i + n3 / 2 : i >= nf3 - n3 / 2 ? i - nf3 + n3 / 2 : -1;
    }
    __device__ __forceinline__ double corr(int iz) const { return den * psi3[iz < n3 / 2 ? n3 / 2 - iz : iz - n3 / 2]; }
    static constexpr bool in_place = false;
    template <int R, int STEP>
    __device__ __forceinline__ void load(int j, Cx<double> (&v)[R], const Cx<double> *__restrict__) const {
        if (m2d) {
#pragma unroll
            for (int q = 0; q < R; ++q) {
                const C<T> *a = in + (j + q * STEP) * plane;
                const C<T> u = ld_once(a, IN_BOUNDS(lim.reads(a, 1), lim.flags));
                v[q] = Cx<double>{(double)u.x, (double)u.y};
            }
        } else {
#pragma unroll
            for (int q = 0; q < R; ++q) {
                const int iz = mode(j + q * STEP);
                const C<T> *a = in + (iz < 0 ? 0 : iz);
                const C<T> u = ld_once(a, iz >= 0 && IN_BOUNDS(lim.reads(a, 1), lim.flags));
                const double w = iz < 0 ? 0.0 : 1.0 / corr(iz);
                v[q] = Cx<double>{(double)u.y * w, (double)u.x * w};      // swapped: the forward direction
            }
        }
    }
    template <int R, int STEP> __device__ __forceinline__ void store(int j, const Cx<double> (&v)[R]) const {
        if (m2d) {
#pragma unroll
            for (int q = 0; q < R; ++q) {
                const int iz = mode(j + q * STEP);
                if (iz < 0 || !IN_BOUNDS(lim.writes(out + iz, 1), lim.flags)) continue;
                const double d = corr(iz);
                out[iz] = C<T>{(T)(v[q].x / d), (T)(v[q].y / d)};
            }
        } else {
#pragma unroll
            for (int q = 0; q < R; ++q) {
                C<T> *o = out + (j + q * STEP) * plane;
                if (IN_BOUNDS(lim.writes(o, 1), lim.flags)) *o = C<T>{(T)v[q].y, (T)v[q].x};
            }
        }
    }
};

template <typename T, class L>
__global__ void __launch_bounds__(L::threads, 512 / L::threads)
k_fft_z(int m2d, DevCorr cc, const Cx<double> *__restrict__ tw, const C<T> *src, C<T> *dst, long long units) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int f = threadIdx.x % L::F, u = threadIdx.x / L::F;
    const int grp = min(u / L::T, L::G - 1), t = u - grp * L::T;
    Cx<double> *sm = reinterpret_cast<Cx<double> *>(smem) + grp * L::pitch * L::F + f;
    const long long want = ((long long)blockIdx.x * L::G + grp) * L::F + f;
    const long long unit = want < units ? want : 0;
    const int xp = (int)(unit / cc.nx), r = (int)(unit - (long long)xp * cc.nx);
    const int r0 = cc.nx - cc.nx / 2, y = r < r0 ? r : r - r0 + cc.nf2 - cc.nx / 2;
    const int ix = r < r0 ? r + cc.nx / 2 : r - r0, kr = r < r0 ? r : cc.nf2 - y;
    const bool right = xp < cc.ny - cc.ny / 2;
    const int ks = right ? xp : cc.ny - xp, iy = right ? xp + cc.ny / 2 : cc.ny / 2 - ks;
    const long long line = (long long)xp * cc.nf2 + y, modes = ((long long)ix * cc.ny + iy) * cc.n3;
    ZMem<T> mem;
    mem.act = t < L::T && want < units;
    mem.m2d = m2d != 0;
    mem.in = src + (m2d ? line : modes);
    mem.out = dst + (m2d ? modes : line);
    mem.plane = (long long)cc.ny * cc.nf2;
    mem.n3 = cc.n3;
    mem.nf3 = L::N;
    const long long nt = mem.plane * L::N, nm = units * cc.n3;
    mem.lim = Limits<T>{src, src + (m2d ? nt : nm), dst, dst + (m2d ? nm : nt), cc.dbg};
    mem.psi3 = cc.psi3;
    mem.den = cc.psi1[ks] * cc.psi2[kr];
    static_for<L::stages>([&](auto k) { fft_stage<L, decltype(k)::v>(t, tw, sm, mem); });
}

}  // namespace curig
