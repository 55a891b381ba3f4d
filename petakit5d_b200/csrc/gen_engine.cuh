// Mixed-radix transform engine for lengths without a compile-time plan: the radices are compile-time
// (straight-line register butterflies), the length, strides and stage order are read at run time from
// a GenAxis table.
//
//  * Lengths whose prime factors are at most 31 run as Stockham stages of the radices below; primes
//    above 5 use the symmetric form of the DFT with the roots as immediates (a quarter of the
//    multiply-adds of the plain sum, no table reads), composites are nested in registers.
//  * Lengths with a larger prime factor keep the in-place engine's sums (stage_direct of fft_engine.cuh).
//
// Stages go from one shared-memory buffer to another, so a stage takes one barrier and its loop is not
// limited by what a thread can hold in registers.  The inverse transform is the forward one on
// swapped re/im, swapped back: the swaps ride on the first load and the last store, and only
// forward butterflies are instantiated.  pass_gen.cuh has the figures of the x / z passes.
#pragma once
#include <type_traits>
#include <utility>

#include "fft_engine.cuh"

namespace pkgen {
using namespace pkfft;

// x / d for x < 2^16, d < 2^16 by one multiply-high: m = floor(2^32 / d) + 1 (d = 1: m = 0, x itself)
struct FastDiv {
    unsigned m;
    __host__ __device__ __forceinline__ explicit FastDiv(unsigned d) : m(d > 1 ? 0xFFFFFFFFu / d + 1u : 0u) {}
    __device__ __forceinline__ int operator()(int x) const { return m ? (int)__umulhi((unsigned)x, m) : x; }
};
__device__ __forceinline__ int fdiv(int x, unsigned m) { return m ? (int)__umulhi((unsigned)x, m) : x; }

// ---- compile-time roots of unity, from the Taylor series in double
constexpr double kPi = 3.14159265358979323846;
constexpr double taylor(double x, int first) {   // first = 0: cos, 1: sin; |x| <= pi
    double t = first ? x : 1.0, s = t;
    for (int k = first + 2; k < 40; k += 2) {
        t *= -x * x / ((double)k * (k - 1));
        s += t;
    }
    return s;
}
// angle 2 pi e / r brought to [-pi, pi]
constexpr double ang(int e, int r) { return 2.0 * kPi * (double)(2 * e > r ? e - r : e) / (double)r; }
template <int E, int R>
constexpr float kCos = (float)taylor(ang(E, R), 0);
template <int E, int R>
constexpr float kSin = (float)taylor(ang(E, R), 1);

template <int... I, class F>
__device__ __forceinline__ void static_for_impl(std::integer_sequence<int, I...>, F&& f) {
    (f(std::integral_constant<int, I>{}), ...);
}
template <int N, class F>
__device__ __forceinline__ void static_for(F&& f) { static_for_impl(std::make_integer_sequence<int, N>{}, f); }

constexpr bool simple_radix(int r) { return r == 2 || r == 3 || r == 4 || r == 5 || r == 8 || r == 16; }
constexpr int radix_a(int r) { return r == 6 ? 2 : r == 9 ? 3 : r == 10 ? 2 : r == 12 ? 4 : r == 15 ? 3 : 0; }

template <int R>
__device__ __forceinline__ void bf_small(float2* v) {
    if constexpr (R == 2) bf2<false>(v[0], v[1]);
    else if constexpr (R == 3) bf3<false>(v);
    else if constexpr (R == 4) bf4<false>(v[0], v[1], v[2], v[3]);
    else if constexpr (R == 5) bf5<false>(v);
    else if constexpr (R == 8) bf8<false>(v);
    else bf16<false>(v);
}

// Forward DFT of odd length R in its symmetric form: with a_m = v_m + v_{R-m}, b_m = v_m - v_{R-m}, X_q and
// X_{R-q} = t1 +- (t2.y, -t2.x) for t1 = v_0 + sum_m a_m cos, t2 = sum_m b_m sin.  emit(q, X[q]) takes each pair
// as it is formed, so R outputs are never held beside the inputs.
template <int R, class E>
__device__ __forceinline__ void bf_odd(float2* v, E&& emit) {
    constexpr int H = (R - 1) / 2;
    float2 a[H], b[H];
    float2 y0 = v[0];
    static_for<H>([&](auto i) {
        a[i.value] = cadd(v[i.value + 1], v[R - 1 - i.value]);
        b[i.value] = csub(v[i.value + 1], v[R - 1 - i.value]);
        y0 = cadd(y0, a[i.value]);
    });
    emit(0, y0);
    static_for<H>([&](auto qi) {
        constexpr int q = qi.value + 1;
        float2 t1 = v[0], t2 = make_float2(0.f, 0.f);
        static_for<H>([&](auto i) {
            constexpr int e = (q * (i.value + 1)) % R;
            t1.x += a[i.value].x * kCos<e, R>;
            t1.y += a[i.value].y * kCos<e, R>;
            t2.x += b[i.value].x * kSin<e, R>;
            t2.y += b[i.value].y * kSin<e, R>;
        });
        emit(q, make_float2(t1.x + t2.y, t1.y - t2.x));
        emit(R - q, make_float2(t1.x - t2.y, t1.y + t2.x));
    });
}

// Forward DFT of R registers; emit(q, X[q]) takes the outputs.
template <int R, class E>
__device__ __forceinline__ void butterfly(float2* v, E&& emit) {
    if constexpr (simple_radix(R)) {
        bf_small<R>(v);
        static_for<R>([&](auto q) { emit(q.value, v[q.value]); });
    } else if constexpr (radix_a(R) > 0) {
        // n = b + B a, k = p + A q: X[p + A q] = sum_b W_B^{b q} W_R^{b p} sum_a v[b + B a] W_A^{a p}
        constexpr int A = radix_a(R), B = R / A;
        float2 t[B][A];
        static_for<B>([&](auto b) {
            static_for<A>([&](auto a) { t[b.value][a.value] = v[b.value + B * a.value]; });
            bf_small<A>(t[b.value]);
        });
        static_for<A>([&](auto p) {
            float2 u[B];
            static_for<B>([&](auto b) {
                constexpr int e = (b.value * p.value) % R;
                const float2 x = t[b.value][p.value];
                if constexpr (e == 0) u[b.value] = x;
                else
                    u[b.value] = make_float2(x.x * kCos<e, R> + x.y * kSin<e, R>, x.y * kCos<e, R> - x.x * kSin<e, R>);
            });
            bf_small<B>(u);
            static_for<B>([&](auto q) { emit(p.value + A * q.value, u[q.value]); });
        });
    } else {
        bf_odd<R>(v, emit);
    }
}

__device__ __forceinline__ float2 swp(float2 a) { return make_float2(a.y, a.x); }

// Table entries of one butterfly's twiddles, rounded up to whole 16-byte pairs.
__host__ __device__ constexpr int tw_row(int R) { return (R - 1 + 1) & ~1; }

// What the first load and the last store of a transform do beside moving the element (block-uniform).
struct GenEdge {
    const float2* otf;       // column tiles: element (l, e) of the OTF at otf[e * es + l], l < ncol
    long long es;
    int ncol, conj;
    int inv;                 // inverse transform: re/im swapped on the way in and out
    float sc;                // factor of the results
};

// Loads of a first stage: as stored; swapped (inverse); * OTF, swapped; any of them, chosen at run time
// (transforms of one stage).  Stores of a last stage: as computed; [swapped,] scaled; either.
enum GenIn { GI_PLAIN, GI_SWAP, GI_OTF, GI_ANY };
enum GenOut { GO_PLAIN, GO_SCALE, GO_ANY };

// Word of element (l, e): column tiles (LF) hold a row of T columns per element, dense as TMA lays it
// out; row tiles hold lines one after the other.  Neither needs spare slots: the first radix is odd, so
// the first stage's stores of consecutive butterflies fall on different banks, and later stages store runs.
template <bool LF>
__device__ __forceinline__ int word(int l, int e, int ls) { return LF ? e * ls + l : l * ls + e; }

// One Stockham stage of radix R over `lines` lines.
template <int R, bool LF, int IN, int OUT>
__device__ __forceinline__ void gstage(const float2* __restrict__ in, float2* __restrict__ out, const GenAxis& A, int s,
                                       int lines, int lt, const GenEdge& g, int kin, int kout, int tid, int nthr) {
    const int m = A.m[s], Ns = A.ns[s];
    const unsigned mg_ns = A.mg_ns[s], mg_m = A.mg_m[s];
    const float2* __restrict__ tw = A.tw + A.off[s];
    const int B = lines * m;
    const int in_kind = IN == GI_ANY ? kin : IN, out_kind = OUT == GO_ANY ? kout : OUT;
    const int ls = LF ? lines : A.n;
    for (int b = tid; b < B; b += nthr) {
        int l, j;
        if constexpr (LF) {
            l = b & (lines - 1);
            j = b >> lt;
        } else {
            l = fdiv(b, mg_m);
            j = b - l * m;
        }
        const int k = Ns > 1 ? j - fdiv(j, mg_ns) * Ns : 0;
        float2 v[R];
        if (in_kind == GI_OTF) {
            // every OTF element is requested before the first is used; columns past the spectrum's
            // (never stored) take the last valid one
            const float2* __restrict__ hp = g.otf + min(l, g.ncol - 1);
#pragma unroll
            for (int r = 0; r < R; r++) v[r] = __ldg(hp + (j + r * m) * g.es);
            const float sg = g.conj ? -1.f : 1.f;
#pragma unroll
            for (int r = 0; r < R; r++)
                v[r] = swp(cmul(in[word<LF>(l, j + r * m, ls)], make_float2(v[r].x, sg * v[r].y)));
        } else {
#pragma unroll
            for (int r = 0; r < R; r++) v[r] = in[word<LF>(l, j + r * m, ls)];
            if (in_kind == GI_SWAP) {
#pragma unroll
                for (int r = 0; r < R; r++) v[r] = swp(v[r]);
            }
        }
        if (Ns > 1) {
            // the butterfly's R - 1 twiddles lie side by side: one address, 16-byte loads
            const float4* __restrict__ tk = reinterpret_cast<const float4*>(tw + k * tw_row(R));
#pragma unroll
            for (int r = 1; r < R; r += 2) {
                const float4 w = __ldg(tk + (r - 1) / 2);
                v[r] = cmul(v[r], make_float2(w.x, w.y));
                if (r + 1 < R) v[r + 1] = cmul(v[r + 1], make_float2(w.z, w.w));
            }
        }
        const int o0 = (j - k) * R + k;
        butterfly<R>(v, [&](int q, float2 x) {
            const int e = o0 + q * Ns;
            if (out_kind == GO_SCALE) {
                if (g.inv) x = swp(x);
                x = make_float2(x.x * g.sc, x.y * g.sc);
            }
            out[word<LF>(l, e, ls)] = x;
        });
    }
}

// Stages by radix.  First stages take an odd radix; BIG adds the radices above 16 (kernels without them run
// with fewer registers).
#define PK_GS_CASE(R, I, O) \
    case R: gstage<R, LF, I, O>(in, out, *A, s, lines, lt, *g, kin, kout, tid, nthr); break;
#define PK_GS_EVEN(I, O) \
    PK_GS_CASE(2, I, O) PK_GS_CASE(4, I, O) PK_GS_CASE(6, I, O) PK_GS_CASE(8, I, O) PK_GS_CASE(10, I, O) \
    PK_GS_CASE(12, I, O) PK_GS_CASE(16, I, O)
#define PK_GS_SMOOTH(I, O) \
    PK_GS_CASE(3, I, O) PK_GS_CASE(5, I, O) PK_GS_CASE(7, I, O) PK_GS_CASE(9, I, O) PK_GS_CASE(15, I, O)
#define PK_GS_MID(I, O) PK_GS_CASE(11, I, O) PK_GS_CASE(13, I, O)
#define PK_GS_BIG(I, O) \
    if constexpr (BIG) switch (rad) { \
        PK_GS_CASE(17, I, O) PK_GS_CASE(19, I, O) PK_GS_CASE(23, I, O) PK_GS_CASE(29, I, O) PK_GS_CASE(31, I, O) \
        default: break; \
    }
#define PK_GS_ARGS \
    const float2 *in, float2 *out, const GenAxis *A, int s, int lines, int lt, const GenEdge *g, int kin, int kout, int tid, \
        int nthr

template <bool LF, bool BIG, int IN>   // first of several stages
__device__ __noinline__ void gs_first(PK_GS_ARGS) {
    const int rad = A->rad[s];
    switch (rad) {
        PK_GS_SMOOTH(IN, GO_PLAIN) PK_GS_MID(IN, GO_PLAIN)
        default: PK_GS_BIG(IN, GO_PLAIN) break;
    }
}
template <bool LF, bool BIG, int OUT>  // middle (OUT = GO_PLAIN) or last of several stages
__device__ __noinline__ void gs_rest(PK_GS_ARGS) {
    const int rad = A->rad[s];
    switch (rad) {
        PK_GS_EVEN(GI_PLAIN, OUT) PK_GS_SMOOTH(GI_PLAIN, OUT) PK_GS_MID(GI_PLAIN, OUT)
        default: PK_GS_BIG(GI_PLAIN, OUT) break;
    }
}
template <bool LF, bool BIG>           // the only stage of a transform
__device__ __noinline__ void gs_only(PK_GS_ARGS) {
    const int rad = A->rad[s];
    switch (rad) {
        PK_GS_SMOOTH(GI_ANY, GO_ANY) PK_GS_MID(GI_ANY, GO_ANY)
        default: PK_GS_BIG(GI_ANY, GO_ANY) break;
    }
}

// Transform of `lines` lines of A.n points from `src` to the buffer returned (b0 or b1; src may be
// either).  `edge` says what the transform's first load (OTF when otf is set) and last store do.  Every
// thread runs before_sync() when it is done with its part of the first stage, and after_first() when the
// whole block is (src may be overwritten then).
template <bool LF, bool BIG, class F0, class F1>
__device__ __forceinline__ float2* gen_transform(const GenAxis* A, const float2* src, float2* b0, float2* b1, int lines,
                                                 int lt, const GenEdge& edge, int tid, int nthr, F0&& before_sync,
                                                 F1&& after_first) {
    const int nst = A->nst;
    const float2* in = src;
    float2* out = src == b0 ? b1 : b0;
    const int kin = LF && edge.otf ? GI_OTF : edge.inv ? GI_SWAP : GI_PLAIN;
    const int kout = edge.inv || edge.sc != 1.f ? GO_SCALE : GO_PLAIN;
    for (int s = 0; s < nst; s++) {
#define PK_GS_CALL(F) F(in, out, A, s, lines, lt, &edge, kin, kout, tid, nthr)
        if (nst == 1) {
            PK_GS_CALL((gs_only<LF, BIG>));
        } else if (s == 0) {
            if (kin == GI_PLAIN) PK_GS_CALL((gs_first<LF, BIG, GI_PLAIN>));
            else if (kin == GI_SWAP) PK_GS_CALL((gs_first<LF, BIG, GI_SWAP>));
            if constexpr (LF) {
                if (kin == GI_OTF) PK_GS_CALL((gs_first<LF, BIG, GI_OTF>));
            }
        } else if (s < nst - 1 || kout == GO_PLAIN) {
            PK_GS_CALL((gs_rest<LF, BIG, GO_PLAIN>));
        } else {
            PK_GS_CALL((gs_rest<LF, BIG, GO_SCALE>));
        }
#undef PK_GS_CALL
        if (s == 0) before_sync();
        __syncthreads();
        if (s == 0) after_first();
        in = out;
        out = out == b0 ? b1 : b0;
    }
    return const_cast<float2*>(in);
}

}  // namespace pkgen
