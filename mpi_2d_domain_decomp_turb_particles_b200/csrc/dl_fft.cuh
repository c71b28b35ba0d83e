// FP64 complex transforms of one line held by a group of threads: Stockham autosort stages
// (Stockham 1966; the radix-R butterflies are compositions of the 2-, 3- and 4-point DFTs by
// the Cooley-Tukey split), each thread keeping its elements of the current stage in
// registers and exchanging them through shared memory between stages.  The flow step
// (dl_flow.cu) builds its passes along z, y and x from this.
#pragma once

#include <cuda_runtime.h>

namespace dlfft {

// A plan: S stages of radix R0, R1, R2 on T threads per line.
template <int N_, int T_, int A, int B, int C = 1>
struct PlanOf {
    static constexpr int N = N_, S = C > 1 ? 3 : 2, T = T_, R0 = A, R1 = B, R2 = C;
};
// Lengths 2^a and 3 * 2^a.  Every stage boundary is a write and a read of the line in shared
// memory, so Wide takes two stages with up to 16 elements per thread, three of 8 beyond 256.  The
// y and z passes run on it everywhere (the transforms alone at 5.6-6.1 TB/s).
template <int N> struct WideT;
template <> struct WideT<32> { using P = PlanOf<32, 4, 8, 4>; };
template <> struct WideT<48> { using P = PlanOf<48, 8, 8, 6>; };
template <> struct WideT<64> { using P = PlanOf<64, 8, 8, 8>; };
template <> struct WideT<96> { using P = PlanOf<96, 8, 12, 8>; };
template <> struct WideT<128> { using P = PlanOf<128, 8, 16, 8>; };
template <> struct WideT<192> { using P = PlanOf<192, 16, 12, 16>; };
template <> struct WideT<256> { using P = PlanOf<256, 16, 16, 16>; };
template <> struct WideT<384> { using P = PlanOf<384, 64, 8, 8, 6>; };
template <> struct WideT<512> { using P = PlanOf<512, 64, 8, 8, 8>; };
// Narrow, for the x pass: from 128 on three stages of 8 elements, with twice Wide's threads per
// line up to 256: the x pass holds six lines per pair of rows in shared memory, which limits the
// threads per SM by lines rather than registers.  Flow step with the droplet field, this and
// Wide: 128^3 203 and 225 us, 192^3 602 and 615, 256^3 1,377 and 1,383.  At 96 the same form takes
// 101.7 us and Wide 99.2.
template <int N> struct NarrowT : WideT<N> {};
template <> struct NarrowT<128> { using P = PlanOf<128, 16, 8, 4, 4>; };
template <> struct NarrowT<192> { using P = PlanOf<192, 32, 8, 8, 3>; };
template <> struct NarrowT<256> { using P = PlanOf<256, 32, 8, 8, 4>; };
template <int N> using Wide = typename WideT<N>::P;
template <int N> using Narrow = typename NarrowT<N>::P;

// Below 32 a tile of 8 kx is half a row and everything is launch latency; above 512 a line needs a
// fourth stage.  Other even sizes would need radices 5, 7, ...
inline bool supported(int n)
{
    switch (n) {
    case 32: case 48: case 64: case 96: case 128: case 192: case 256: case 384: case 512: return true;
    default: return false;
    }
}

__host__ __device__ constexpr int div_up(int a, int b) { return (a + b - 1) / b; }

// stage geometry: NB butterflies of radix R, NS = product of the earlier radices, NI
// butterflies per thread, table offset of its twiddles
template <class P, int s>
struct Stage {
    static constexpr int R = s == 0 ? P::R0 : (s == 1 ? P::R1 : P::R2), NB = P::N / R;
    static constexpr int NS = s == 0 ? 1 : (s == 1 ? P::R0 : P::R0 * P::R1);
    static constexpr int NI = div_up(NB, P::T);
    static constexpr bool FULL = NB % P::T == 0;   // every thread has NI butterflies
    static constexpr int TW = s <= 1 ? 0 : (P::R1 - 1) * P::R0;
};
// elements a thread holds in the widest stage
template <class P>
__host__ __device__ constexpr int elems()
{
    int e = Stage<P, 0>::NI * Stage<P, 0>::R;
    if (Stage<P, 1>::NI * Stage<P, 1>::R > e) e = Stage<P, 1>::NI * Stage<P, 1>::R;
    if (P::S > 2 && div_up(P::N / P::R2, P::T) * P::R2 > e)
        e = div_up(P::N / P::R2, P::T) * P::R2;
    return e;
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
// a * (c + i SIGN s)
template <int SIGN>
__device__ __forceinline__ double2 cmulw(double2 a, double c, double s)
{
    if (SIGN > 0) return make_double2(fma(a.x, c, -(a.y * s)), fma(a.y, c, a.x * s));
    return make_double2(fma(a.x, c, a.y * s), fma(a.y, c, -(a.x * s)));
}
// a * (SIGN i)
template <int SIGN>
__device__ __forceinline__ double2 cmuli(double2 a)
{
    return SIGN > 0 ? make_double2(-a.y, a.x) : make_double2(a.y, -a.x);
}

// cos and sin of 2 pi e / 48 for the butterflies' inner twiddles (R = 6, 8, 12, 16)
__host__ __device__ constexpr double cos48(int e)
{
    e = ((e % 48) + 48) % 48;
    if (e > 24) e = 48 - e;
    const bool neg = e > 12;
    if (neg) e = 24 - e;
    double v = 0.0;
    switch (e) {
    case 0: v = 1.0; break;
    case 1: v = 0.99144486137381041114; break;
    case 2: v = 0.96592582628906828675; break;
    case 3: v = 0.92387953251128675613; break;
    case 4: v = 0.86602540378443864676; break;
    case 5: v = 0.79335334029123516458; break;
    case 6: v = 0.70710678118654752440; break;
    case 7: v = 0.60876142900872063942; break;
    case 8: v = 0.5; break;
    case 9: v = 0.38268343236508977173; break;
    case 10: v = 0.25881904510252076235; break;
    case 11: v = 0.13052619222005159155; break;
    default: v = 0.0; break;
    }
    return neg ? -v : v;
}
__host__ __device__ constexpr double sin48(int e) { return cos48(12 - e); }

// a * exp(SIGN 2 pi i E / 48), E a compile-time constant
template <int SIGN, int E>
__device__ __forceinline__ double2 rot48(double2 a)
{
    constexpr int e = ((E % 48) + 48) % 48;
    constexpr double c = cos48(e), s = sin48(e);
    if constexpr (e == 0) return a;
    else if constexpr (e == 24) return make_double2(-a.x, -a.y);
    else if constexpr (e == 12) return cmuli<SIGN>(a);
    else if constexpr (e == 36) return cmuli<-SIGN>(a);
    else if constexpr (e == 6 || e == 18 || e == 30 || e == 42) {
        // (+-1 +- i) sqrt(1/2): two additions and two products
        constexpr double h = 0.70710678118654752440;
        constexpr double cs = c > 0 ? h : -h, ss = (s > 0) == (SIGN > 0) ? h : -h;
        return make_double2(cs * a.x - ss * a.y, cs * a.y + ss * a.x);
    } else return cmulw<SIGN>(a, c, s);
}

template <int SIGN, int R>
struct Dft;
template <int SIGN>
struct Dft<SIGN, 2> {
    static __device__ __forceinline__ void run(double2 *v)
    {
        const double2 a = v[0], b = v[1];
        v[0] = cadd(a, b);
        v[1] = csub(a, b);
    }
};
template <int SIGN>
struct Dft<SIGN, 3> {
    static __device__ __forceinline__ void run(double2 *v)
    {
        const double2 s = cadd(v[1], v[2]), d = cmuli<SIGN>(csub(v[1], v[2]));
        const double2 m = make_double2(fma(-0.5, s.x, v[0].x), fma(-0.5, s.y, v[0].y));
        constexpr double h = 0.86602540378443864676;
        v[0] = cadd(v[0], s);
        v[1] = make_double2(fma(h, d.x, m.x), fma(h, d.y, m.y));
        v[2] = make_double2(fma(-h, d.x, m.x), fma(-h, d.y, m.y));
    }
};
template <int SIGN>
struct Dft<SIGN, 4> {
    static __device__ __forceinline__ void run(double2 *v)
    {
        const double2 a = cadd(v[0], v[2]), b = csub(v[0], v[2]);
        const double2 c = cadd(v[1], v[3]), d = cmuli<SIGN>(csub(v[1], v[3]));
        v[0] = cadd(a, c);
        v[1] = cadd(b, d);
        v[2] = csub(a, c);
        v[3] = csub(b, d);
    }
};
// R = A * B: A-point transforms over the stride-B subsequences, rotations, B-point transforms
template <int SIGN, int A, int B>
struct DftAB {
    template <int n2, int k1>
    static __device__ __forceinline__ void rot(double2 *w)
    {
        if constexpr (k1 < A) {
            w[k1] = rot48<SIGN, n2 * k1 * (48 / (A * B))>(w[k1]);
            rot<n2, k1 + 1>(w);
        }
    }
    template <int n2>
    static __device__ __forceinline__ void first(const double2 *v, double2 (*y)[A])
    {
        if constexpr (n2 < B) {
            double2 w[A];
#pragma unroll
            for (int n1 = 0; n1 < A; n1++) w[n1] = v[B * n1 + n2];
            Dft<SIGN, A>::run(w);
            rot<n2, 1>(w);
#pragma unroll
            for (int k = 0; k < A; k++) y[n2][k] = w[k];
            first<n2 + 1>(v, y);
        }
    }
    static __device__ __forceinline__ void run(double2 *v)
    {
        double2 y[B][A];
        first<0>(v, y);
#pragma unroll
        for (int k1 = 0; k1 < A; k1++) {
            double2 w[B];
#pragma unroll
            for (int n2 = 0; n2 < B; n2++) w[n2] = y[n2][k1];
            Dft<SIGN, B>::run(w);
#pragma unroll
            for (int k2 = 0; k2 < B; k2++) v[k1 + A * k2] = w[k2];
        }
    }
};
template <int SIGN> struct Dft<SIGN, 6> : DftAB<SIGN, 2, 3> {};
template <int SIGN> struct Dft<SIGN, 8> : DftAB<SIGN, 4, 2> {};
template <int SIGN> struct Dft<SIGN, 12> : DftAB<SIGN, 4, 3> {};
template <int SIGN> struct Dft<SIGN, 16> : DftAB<SIGN, 4, 4> {};

// Index of the element v[i * R + m] that thread t holds at the input and at the output of
// stage s; in_at also serves the line's input (s = 0) and out_at its result (s = S - 1).
template <class P, int s>
__device__ __forceinline__ int in_at(int t, int i, int m)
{
    return t + P::T * i + m * Stage<P, s>::NB;
}
template <class P, int s>
__device__ __forceinline__ int out_at(int t, int i, int m)
{
    constexpr int NS = Stage<P, s>::NS, R = Stage<P, s>::R;
    const int b = t + P::T * i;
    if constexpr (s == 0) return b * R + m;
    else return (b / NS) * (NS * R) + b % NS + m * NS;
}
template <class P, int s>
__device__ __forceinline__ bool has(int t, int i)
{
    return Stage<P, s>::FULL || t + P::T * i < Stage<P, s>::NB;
}
// f(i, m) for the elements a thread holds at stage s
template <class P, int s, typename F>
__device__ __forceinline__ void each(int t, F f)
{
#pragma unroll
    for (int i = 0; i < Stage<P, s>::NI; i++)
        if (has<P, s>(t, i)) {
#pragma unroll
            for (int m = 0; m < Stage<P, s>::R; m++) f(i, m);
        }
}

// tw: for each stage after the first, w^(m q) at (m - 1) * NS + q (contiguous in q, the
// index neighbouring threads differ in).  Reading a quarter of the powers and multiplying the
// rest from them was no faster in any pass (x at 256^3, in two stages: 0.58 against 0.49 ms).
template <class P, int SIGN, int s>
__device__ __forceinline__ void butterflies(int t, double2 *v, const double2 *__restrict__ tw)
{
    using St = Stage<P, s>;
#pragma unroll
    for (int i = 0; i < St::NI; i++) {
        if (!has<P, s>(t, i)) continue;
        if constexpr (s > 0) {
            const int q = (t + P::T * i) % St::NS;
#pragma unroll
            for (int m = 1; m < St::R; m++) {
                const double2 w = __ldg(tw + St::TW + (m - 1) * St::NS + q);
                v[i * St::R + m] = cmulw<SIGN>(v[i * St::R + m], w.x, w.y);
            }
        }
        Dft<SIGN, St::R>::run(v + i * St::R);
    }
}

// One line: v holds the input elements of stage 0 and returns those of the last stage's
// output (unnormalised, exp(SIGN 2 pi i k x / N)).  `at` maps a line index to this line's
// slot in `buf`; `sync` is a barrier of (at least) the threads of the line, which all call
// this.  The buffer is free to be overwritten on entry, and after the next barrier on return.
template <class P, int SIGN, typename At, typename Sync>
__device__ __forceinline__ void line(int t, double2 *v, double2 *buf, At at, const double2 *__restrict__ tw, Sync sync)
{
    butterflies<P, SIGN, 0>(t, v, tw);
    each<P, 0>(t, [&](int i, int m) { buf[at(out_at<P, 0>(t, i, m))] = v[i * Stage<P, 0>::R + m]; });
    sync();
    each<P, 1>(t, [&](int i, int m) { v[i * Stage<P, 1>::R + m] = buf[at(in_at<P, 1>(t, i, m))]; });
    butterflies<P, SIGN, 1>(t, v, tw);
    if constexpr (P::S > 2) {
        sync();
        each<P, 1>(t, [&](int i, int m) { buf[at(out_at<P, 1>(t, i, m))] = v[i * Stage<P, 1>::R + m]; });
        sync();
        each<P, 2>(t, [&](int i, int m) { v[i * Stage<P, 2>::R + m] = buf[at(in_at<P, 2>(t, i, m))]; });
        butterflies<P, SIGN, 2>(t, v, tw);
    }
}
struct BlockSync {
    __device__ __forceinline__ void operator()() const { __syncthreads(); }
};
// the threads of one line of a block whose lines are groups of T consecutive threads
template <int T>
struct LineSync {
    int id;   // line within the block
    __device__ __forceinline__ void operator()() const
    {
        if constexpr (T <= 32) __syncwarp();
        else asm volatile("bar.sync %0, %1;" ::"r"(id + 1), "n"(T) : "memory");
    }
};

}  // namespace dlfft
