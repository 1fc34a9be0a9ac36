// fft_core.cuh -- building blocks of the batched line FFTs of the RK3 step (FP64
// and FP32).
//
// The reference runs FFTW 1-D plans (src/pf_fftw.f90:199-291): c2c along z and y,
// c2r/r2c along x, FFTW_BACKWARD (e^{+2 pi i kn/N}) unnormalised for
// spectral->physical and FFTW_FORWARD (e^{-2 pi i kn/N}) for physical->spectral.
// Here the same transforms are radix-R Stockham autosort passes (the formulation
// of Govindaraju et al., "High performance discrete Fourier transforms on
// graphics processors", SC 2008) over a tile of L lines held in shared memory
// in column layout: element n of line l sits at s[n*LP + l] (LP >= L, odd pad
// so that the transposing global<->shared copies are bank-conflict free).
// Each pass: load R points of stride N/R, twiddle by W_{Ns R}^{r k}, R-point DFT
// in registers, store at (j/Ns)*Ns*R + j%Ns + r*Ns.
//
// Everything here is __host__ __device__ so that the index arithmetic and the
// small DFTs are exercised on the CPU by the unit test harness (fft_core_test.cpp)
// before they run on a GPU.
#pragma once

#if defined(__CUDACC__)
#include <cuda_runtime.h>
#define PD_HD __host__ __device__ __forceinline__
#else
#include <cstddef>
struct double2 { double x, y; };
struct float2 { float x, y; };
#define PD_HD inline
#endif

namespace pdfft {

// Complex values are double2 (the FP64 form) or float2 (the FP32-mixed form);
// every helper below is generic over the two, the real type following the
// arguments.  Constants are written in FP64 and rounded once to the real type.
template <class T> struct cplx;
template <> struct cplx<double> { using type = double2; };
template <> struct cplx<float> { using type = float2; };
template <class C> using real_of = decltype(C{}.x);

PD_HD double2 mk(double x, double y) { double2 r; r.x = x; r.y = y; return r; }
PD_HD float2 mk(float x, float y) { float2 r; r.x = x; r.y = y; return r; }
// On sm_100 the FP32 form issues its complex arithmetic as packed two-lane FP32
// instructions (__fadd2_rn, __fmul2_rn, __ffma2_rn: per component the same
// rounding as the scalar operation), which halves the instruction count of the
// butterflies.  PD_F32X2 is the device pass for such a target.
#if defined(__CUDA_ARCH__) && (__CUDA_ARCH__ >= 1000)
#define PD_F32X2 1
#else
#define PD_F32X2 0
#endif
template <class A, class B> struct same_type { static constexpr bool value = false; };
template <class A> struct same_type<A, A> { static constexpr bool value = true; };
template <class C> constexpr bool packed_f32() { return PD_F32X2 && same_type<C, float2>::value; }

template <class C> PD_HD C add(C a, C b) {
#if PD_F32X2
    if constexpr (packed_f32<C>()) return __fadd2_rn(a, b);
    else
#endif
    return mk(a.x + b.x, a.y + b.y);
}
template <class C> PD_HD C sub(C a, C b) {
#if PD_F32X2
    if constexpr (packed_f32<C>()) return __fadd2_rn(a, mk(-b.x, -b.y));
    else
#endif
    return mk(a.x - b.x, a.y - b.y);
}
template <class C> PD_HD C scl(C a, double s) {
    const real_of<C> t = (real_of<C>)s;
#if PD_F32X2
    if constexpr (packed_f32<C>()) return __fmul2_rn(a, mk(t, t));
    else
#endif
    return mk(a.x * t, a.y * t);
}
// a * b = (a.x, a.x) * b + (a.y, a.y) * (-b.y, b.x)
template <class C> PD_HD C cmul(C a, C b) {
#if PD_F32X2
    if constexpr (packed_f32<C>()) return __ffma2_rn(mk(a.x, a.x), b, __fmul2_rn(mk(a.y, a.y), mk(-b.y, b.x)));
    else
#endif
    return mk(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// a * conj(b) = a * (b.x, b.x) + (a.y, -a.x) * (b.y, b.y)
template <class C> PD_HD C cmulc(C a, C b) {
#if PD_F32X2
    if constexpr (packed_f32<C>()) return __ffma2_rn(a, mk(b.x, b.x), __fmul2_rn(mk(a.y, -a.x), mk(b.y, b.y)));
    else
#endif
    return mk(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}

// Sign convention: a DFT of sign S computes X_r = sum_q x_q exp(S * 2 pi i q r / R);
// S = -1 is FFTW_FORWARD, S = +1 is FFTW_BACKWARD.  Twiddle tables hold
// tw[e] = exp(-2 pi i e / N); a sign-S pass multiplies by tw (S=-1) or conj(tw).
template <int S, class C> PD_HD C twmul(C a, C w) { return S < 0 ? cmul(a, w) : cmulc(a, w); }
// a * (S i)
template <int S, class C> PD_HD C mul_si(C a) { return S > 0 ? mk(-a.y, a.x) : mk(a.y, -a.x); }
// a + k b for a real constant k
template <class C> PD_HD C axpy(C a, double k, C b) {
    const real_of<C> t = (real_of<C>)k;
#if PD_F32X2
    if constexpr (packed_f32<C>()) return __ffma2_rn(mk(t, t), b, a);
    else
#endif
    return mk(a.x + t * b.x, a.y + t * b.y);
}
// The butterfly of a constant twiddle w = c + S i s: p = e + w o, m = e - w o, with the
// larger of c and s taken out of w, so that the product of the twiddle and the two sums are
// six fused multiply-adds (a complex product and two sums: four and four).  In the FP64 x pass,
// bound by its FP64 instructions at 8 to 16 warps per SM, this, the zero inputs of truncated
// spectra (below), the shared twiddles of wpass_n and one-warp CTAs took the 512-point pass of
// 512^3 from 2.99 to 2.52 ms per stage, the 256-point one from 0.334 to 0.312, the R-conv one
// at 192^3 from 0.445 to 0.306 (FP32-mixed at 512^3: 1.46 to 1.28).
template <int S, class C> PD_HD void bfly_cs(C e, C o, double c, double s, C& p, C& m) {
    const double cs = S * s;
    const bool cl = (c < 0 ? -c : c) >= (s < 0 ? -s : s);   // folded: c and s are literals
    const C io = mk(-o.y, o.x);
    const C q = cl ? axpy(o, cs / c, io) : axpy(io, c / cs, o);
    const double f = cl ? c : cs;
    p = axpy(e, f, q);
    m = axpy(e, -f, q);
}
// p = a + b, m = a - b, where ZA / ZB say that a / b is a zero known at compile time (an
// input outside the band of a truncated spectrum): no arithmetic is spent on it.
template <bool ZA, bool ZB, class C> PD_HD void addsub(C a, C b, C& p, C& m) {
    if constexpr (ZB) { p = a; m = a; }
    else if constexpr (ZA) { p = b; m = mk(-b.x, -b.y); }
    else { p = add(a, b); m = sub(a, b); }
}
// The even / odd bits of an input mask.
constexpr unsigned even_bits(unsigned z) {
    unsigned r = 0;
    for (int q = 0; q < 16; q++) r |= ((z >> (2 * q)) & 1u) << q;
    return r;
}
constexpr unsigned odd_bits(unsigned z) { return even_bits(z >> 1); }

constexpr double kSqrtHalf = 0.7071067811865475244008444;
constexpr double kSin60 = 0.8660254037844386467637232;

// DFTs of 2..32 points in registers (2, 3, 4, 5, 7, 8, 10, 12, 14, 16, 20, 24, 28, 32).  Z: mask
// of the inputs that are zero at compile time.
template <int S, unsigned Z = 0, class C> PD_HD void dft2(C* v) {
    C a = v[0], b = v[1];
    addsub<(Z & 1u) != 0, (Z & 2u) != 0>(a, b, v[0], v[1]);
}
template <int S, class C> PD_HD void dft3(C* v) {
    const C t = add(v[1], v[2]), d = mul_si<S>(sub(v[1], v[2]));
    const C m = axpy(v[0], -0.5, t);
    v[0] = add(v[0], t);
    v[1] = axpy(m, kSin60, d);
    v[2] = axpy(m, -kSin60, d);
}
template <int S, unsigned Z = 0, class C> PD_HD void dft4(C* v) {
    C a0, a1, b0, b1;
    addsub<(Z & 1u) != 0, (Z & 4u) != 0>(v[0], v[2], a0, a1);
    addsub<(Z & 2u) != 0, (Z & 8u) != 0>(v[1], v[3], b0, b1);
    b1 = mul_si<S>(b1);
    v[0] = add(a0, b0); v[2] = sub(a0, b0);
    v[1] = add(a1, b1); v[3] = sub(a1, b1);
}
template <int S, unsigned Z = 0, class C> PD_HD void dft8(C* v) {
    C e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
    dft4<S, even_bits(Z)>(e); dft4<S, odd_bits(Z)>(o);
    o[2] = mul_si<S>(o[2]);
    v[0] = add(e[0], o[0]); v[4] = sub(e[0], o[0]);
    bfly_cs<S>(e[1], o[1], kSqrtHalf, kSqrtHalf, v[1], v[5]);
    v[2] = add(e[2], o[2]); v[6] = sub(e[2], o[2]);
    bfly_cs<S>(e[3], o[3], -kSqrtHalf, kSqrtHalf, v[3], v[7]);
}
// cos and sin of pi r / 16, r = 0..8 (sin of r is cos of 8 - r)
PD_HD double cos16(int r) {
    return r == 0 ? 1.0 : r == 1 ? 0.9807852804032304491261822 : r == 2 ? 0.9238795325112867561281832
         : r == 3 ? 0.8314696123025452370787884 : r == 4 ? kSqrtHalf : r == 5 ? 0.5555702330196022247428308
         : r == 6 ? 0.38268343236508977172846 : r == 7 ? 0.1950903220161282678482849 : 0.0;
}
// Twiddle W_{2H}^(S r) = cos(pi r / H) + S i sin(pi r / H), H = 8 or 16, applied in the last
// radix-2 step of an even/odd split: v[r], v[r + H] = e[r] +- w o[r].
template <int S, int H, class C> PD_HD void combine(const C* e, const C* o, C* v) {
    constexpr int q = 16 / H;   // units of pi / 16
#pragma unroll
    for (int r = 0; r < H; r++) {
        if (r == 0) { v[0] = add(e[0], o[0]); v[H] = sub(e[0], o[0]); }
        else if (2 * r == H) {
            const C t = mul_si<S>(o[r]);
            v[r] = add(e[r], t); v[r + H] = sub(e[r], t);
        } else {
            const double c = 2 * r < H ? cos16(q * r) : -cos16(16 - q * r);
            const double s = 2 * r < H ? cos16(8 - q * r) : cos16(q * r - 8);
            bfly_cs<S>(e[r], o[r], c, s, v[r], v[r + H]);
        }
    }
}
template <int S, unsigned Z = 0, class C> PD_HD void dft16(C* v) {
    C e[8], o[8];
#pragma unroll
    for (int q = 0; q < 8; q++) { e[q] = v[2 * q]; o[q] = v[2 * q + 1]; }
    dft8<S, even_bits(Z)>(e); dft8<S, odd_bits(Z)>(o);
    combine<S, 8>(e, o, v);
}
// 32 = 2 x 16: radix-2 decimation in time over two length-16 DFTs.
template <int S, unsigned Z = 0, class C> PD_HD void dft32(C* v) {
    C e[16], o[16];
#pragma unroll
    for (int q = 0; q < 16; q++) { e[q] = v[2 * q]; o[q] = v[2 * q + 1]; }
    dft16<S, even_bits(Z)>(e); dft16<S, odd_bits(Z)>(o);
    combine<S, 16>(e, o, v);
}
// 12 = 3 x 4 (Cooley-Tukey): n = 4 n1 + n2, k = k1 + 3 k2.  Length-3 DFTs over n1
// for each n2, twiddles W12^(S n2 k1) (multiples of 30 degrees) folded into the first
// butterflies of the length-4 DFTs over n2 for each k1.
template <int S, class C> PD_HD void dft12(C* v) {
    C y[4][3];
#pragma unroll
    for (int n2 = 0; n2 < 4; n2++) {
        y[n2][0] = v[n2]; y[n2][1] = v[4 + n2]; y[n2][2] = v[8 + n2];
        dft3<S>(y[n2]);
    }
    C z[4] = {y[0][0], y[1][0], y[2][0], y[3][0]};
    dft4<S>(z);
#pragma unroll
    for (int k2 = 0; k2 < 4; k2++) v[3 * k2] = z[k2];
    C a0, a1, p, m;
    // k1 = 1: twiddles 30, 60 and 90 degrees; p, m = i S y3 +- w1 y1
    bfly_cs<S>(y[0][1], y[2][1], 0.5, kSin60, a0, a1);
    bfly_cs<S>(mul_si<S>(y[3][1]), y[1][1], kSin60, 0.5, p, m);
    m = mul_si<S>(m);
    v[1] = add(a0, p); v[7] = sub(a0, p);
    v[4] = sub(a1, m); v[10] = add(a1, m);
    // k1 = 2: twiddles 60, 120 and 180 degrees; p, m = y3 +- w1 y1
    bfly_cs<S>(y[0][2], y[2][2], -0.5, kSin60, a0, a1);
    bfly_cs<S>(y[3][2], y[1][2], 0.5, kSin60, p, m);
    p = mul_si<S>(p);
    v[2] = sub(a0, m); v[8] = add(a0, m);
    v[5] = add(a1, p); v[11] = sub(a1, p);
}
// odd prime R (5, 7): X_r, X_{R-r} = A_r +- S i B_r with A_r = v0 + sum_q C(qr)(v_q + v_{R-q}),
// B_r = sum_q S(qr)(v_q - v_{R-q}), q = 1..(R-1)/2
template <int R> struct PrimeTab;
template <> struct PrimeTab<5> {
    static PD_HD double c(int m) {
        return m == 0 ? 1.0 : (m == 1 || m == 4) ? 0.3090169943749474241022934 : -0.8090169943749474241022934;
    }
    static PD_HD double s(int m) {
        return m == 0 ? 0.0 : m == 1 ? 0.9510565162951535721164393 : m == 2 ? 0.587785252292473129168706
             : m == 3 ? -0.587785252292473129168706 : -0.9510565162951535721164393;
    }
};
template <> struct PrimeTab<7> {
    static PD_HD double c(int m) {
        return m == 0 ? 1.0 : (m == 1 || m == 6) ? 0.6234898018587335305250049
             : (m == 2 || m == 5) ? -0.2225209339563144042889026 : -0.9009688679024191262361023;
    }
    static PD_HD double s(int m) {
        return m == 0 ? 0.0 : m == 1 ? 0.7818314824680298087084445 : m == 2 ? 0.9749279121818236070181317
             : m == 3 ? 0.4338837391175581204757683 : m == 4 ? -0.4338837391175581204757683
             : m == 5 ? -0.9749279121818236070181317 : -0.7818314824680298087084445;
    }
};
template <int R, int S, unsigned Z = 0, class C> PD_HD void dft_prime(C* v) {
    constexpr int H = (R - 1) / 2;
    // the one input that can be zero at compile time: the middle one, v_H (pair H, H + 1)
    constexpr bool zm = ((Z >> H) & 1u) != 0;
    static_assert((Z & ~(1u << H)) == 0, "zero mask of a prime radix");
    C sum[H], dif[H];
#pragma unroll
    for (int q = 1; q <= H; q++) {
        if (q == H) addsub<zm, false>(v[q], v[R - q], sum[q - 1], dif[q - 1]);
        else addsub<false, false>(v[q], v[R - q], sum[q - 1], dif[q - 1]);
        dif[q - 1] = mul_si<S>(dif[q - 1]);
    }
    const C x0 = v[0];
    C t = x0;
#pragma unroll
    for (int q = 0; q < H; q++) t = add(t, sum[q]);
    v[0] = t;
#pragma unroll
    for (int r = 1; r <= H; r++) {
        C a = x0, b = scl(dif[0], PrimeTab<R>::s(r));
#pragma unroll
        for (int q = 1; q <= H; q++) {
            const int m = (q * r) % R;
            a = axpy(a, PrimeTab<R>::c(m), sum[q - 1]);
            if (q > 1) b = axpy(b, PrimeTab<R>::s(m), dif[q - 1]);
        }
        v[r] = add(a, b);
        v[R - r] = sub(a, b);
    }
}

// R = P Q with P = 2, 4 or 8 and Q = 3, 5 or 7, without twiddles (the prime-factor mapping of
// Good, 1958): with n = Q n1 + P n2 mod R the kernel splits into exp(2 pi i n1 k / P) exp(2 pi i n2 k / Q), so
// P-point DFTs over n1 and Q-point DFTs over n2 give X_k for k = k1 mod P, k = k2 mod Q.
template <int I, int N, class F> PD_HD void for_range(F& f);
template <int I> struct Ix { static constexpr int value = I; };
template <int I, int N, class F> PD_HD void for_range(F& f) {
    if constexpr (I < N) {
        f(Ix<I>{});
        for_range<I + 1, N>(f);
    }
}
template <int P, int Q> constexpr int crt(int k1, int k2) {
    for (int k = 0; k < P * Q; k++)
        if (k % P == k1 && k % Q == k2) return k;
    return -1;
}
template <int P, int Q> constexpr unsigned pfa_mask(unsigned z, int n2) {
    unsigned r = 0;
    for (int n1 = 0; n1 < P; n1++) r |= ((z >> ((Q * n1 + P * n2) % (P * Q))) & 1u) << n1;
    return r;
}
template <int P, int Q, int S, unsigned Z = 0, class C> PD_HD void dft_pfa(C* v) {
    C y[P][Q];
    auto rows = [&](auto ix) {
        constexpr int n2 = decltype(ix)::value;
        C t[P];
#pragma unroll
        for (int n1 = 0; n1 < P; n1++) t[n1] = v[(Q * n1 + P * n2) % (P * Q)];
        if constexpr (P == 2) dft2<S, pfa_mask<P, Q>(Z, n2)>(t);
        else if constexpr (P == 4) dft4<S, pfa_mask<P, Q>(Z, n2)>(t);
        else dft8<S, pfa_mask<P, Q>(Z, n2)>(t);
#pragma unroll
        for (int n1 = 0; n1 < P; n1++) y[n1][n2] = t[n1];
    };
    for_range<0, Q>(rows);
    auto cols = [&](auto ix) {
        constexpr int k1 = decltype(ix)::value;
        if constexpr (Q == 3) dft3<S>(y[k1]);
        else dft_prime<Q, S>(y[k1]);
        auto put = [&](auto iy) {
            constexpr int k2 = decltype(iy)::value, k = crt<P, Q>(k1, k2);
            v[k] = y[k1][k2];
        };
        for_range<0, Q>(put);
    };
    for_range<0, P>(cols);
}

template <int R, int S, unsigned Z = 0, class C> PD_HD void dft(C* v) {
    if constexpr (R == 2) dft2<S, Z>(v);
    else if constexpr (R == 3) dft3<S>(v);
    else if constexpr (R == 4) dft4<S, Z>(v);
    else if constexpr (R == 8) dft8<S, Z>(v);
    else if constexpr (R == 16) dft16<S, Z>(v);
    else if constexpr (R == 12) dft12<S>(v);
    else if constexpr (R == 32) dft32<S, Z>(v);
    else if constexpr (R == 5 || R == 7) dft_prime<R, S, Z>(v);
    else if constexpr (R == 10) dft_pfa<2, 5, S, Z>(v);
    else if constexpr (R == 14) dft_pfa<2, 7, S, Z>(v);
    else if constexpr (R == 20) dft_pfa<4, 5, S, Z>(v);
    else if constexpr (R == 24) dft_pfa<8, 3, S, Z>(v);
    else if constexpr (R == 28) dft_pfa<4, 7, S, Z>(v);
    else static_assert(R == 2, "unsupported radix");
}

// Radix schedule per transform length.  Supported N: 2^a * {1,3,5,7} from 16 to 1024,
// factored into at most three radices.  Composite radices with a factor 3, 5 or 7 where they save
// a pass, each a shared-memory round trip and a barrier: two passes against three took the shear
// step of 160^3 from 0.819 to 0.659 ms (FP32-mixed 0.452 -> 0.377), 224^3 2.02 -> 1.64 (1.28 ->
// 0.91), 320^3 5.49 -> 4.99 (3.30 -> 2.72), 384^3 12.1 -> 9.32 (6.23 -> 4.66).
template <int N> struct Plan { static constexpr int r0 = 0, r1 = 0, r2 = 0; };
#define PD_PLAN(N_, A, B, C) \
    template <> struct Plan<N_> { static constexpr int r0 = A, r1 = B, r2 = C; };
PD_PLAN(16, 16, 0, 0)
PD_PLAN(24, 3, 8, 0)
PD_PLAN(32, 8, 4, 0)
PD_PLAN(40, 5, 8, 0)
PD_PLAN(48, 3, 16, 0)
PD_PLAN(56, 7, 8, 0)
PD_PLAN(64, 8, 8, 0)
PD_PLAN(80, 5, 16, 0)
PD_PLAN(96, 8, 12, 0)
PD_PLAN(112, 7, 16, 0)
PD_PLAN(128, 8, 16, 0)
PD_PLAN(160, 10, 16, 0)
PD_PLAN(192, 16, 12, 0)
PD_PLAN(224, 14, 16, 0)
PD_PLAN(256, 16, 16, 0)
PD_PLAN(320, 20, 16, 0)
PD_PLAN(384, 24, 16, 0)
PD_PLAN(448, 7, 8, 8)
PD_PLAN(512, 8, 8, 8)
PD_PLAN(640, 5, 8, 16)
PD_PLAN(768, 3, 16, 16)
PD_PLAN(896, 7, 8, 16)
PD_PLAN(1024, 16, 8, 8)
#undef PD_PLAN

template <int N> constexpr bool plan_ok() {
    return Plan<N>::r0 * (Plan<N>::r1 ? Plan<N>::r1 : 1) * (Plan<N>::r2 ? Plan<N>::r2 : 1) == N;
}

// Row of element n in a tile: with PS = a > 0 one pad row follows every 2^a rows, with
// PS = a + 16 b another every 2^b rows, which spreads the stores of the passes, of stride the
// radix, over distinct banks when a warp owns whole lines.  (Shifts of n, not an exclusive-or
// swizzle: n = j + r N / R then keeps a compile-time offset per r.)
template <int PS> PD_HD constexpr int prow(int n) {
    return PS <= 0 ? n : (PS < 16 ? n + (n >> PS) : n + (n >> (PS & 15)) + (n >> (PS >> 4)));
}
template <int N, int PS> constexpr int tile_rows() { return prow<PS>(N - 1) + 1; }

// One pass, split into a load/compute half and a store half so that a CPU
// emulator can run all items' first halves before any second half (that is
// what the __syncthreads() between them does on the GPU).
// Element n of line l: interleaved columns (AS = 0, s[prow(n)*LP + l]) or separate
// arrays AS elements apart (s[l*AS + prow(n)]).
template <int LP, int PS, int AS> PD_HD int tidx(int n, int l) {
    return AS ? l * AS + prow<PS>(n) : prow<PS>(n) * LP + l;
}

// Line and index of item w of a pass with NR items per line: the lines of a tile interleave
// (neighbouring items are one butterfly of neighbouring lines); separate arrays that share a
// warp's lanes (NR <= 16) follow one another, so that the lanes of a wavefront stay in one.
template <int NR, int L, int AS> PD_HD int item_line(int w) { return AS && NR <= 16 ? w / NR : w % L; }
template <int NR, int L, int AS> PD_HD int item_index(int w) { return AS && NR <= 16 ? w % NR : w / L; }

// Twiddles w[r] = tw[r e] (r = 1..R-1) of one butterfly: the entries at power-of-two
// multiples r = 2^a are read from the table (log2 R loads), the others are products
// w[2^a] w[r - 2^a] of those (at most log2(R) - 1 roundings on a correctly rounded
// entry).  The kernels are bound by load instructions and shared/L1 wavefronts, so
// the table reads are what is saved; the FP arithmetic has room.
template <int R, class C> PD_HD void twiddles(const C* tw, int e, C* w) {
#pragma unroll
    for (int r = 1; r < R; r++) {
        if ((r & (r - 1)) == 0) {
            w[r] = tw[r * e];
        } else {
            int hb = 1;
            while (hb * 2 <= r) hb *= 2;
            w[r] = cmul(w[hb], w[r - hb]);
        }
    }
}

// The band of a 2/3-truncated spectrum on a length-N line: n <= KB or n >= N - KB
// (KB = 0: the whole line).  A pass_load with KB > 0 reads the elements outside
// the band as zero without touching shared memory (first pass of a transform of a
// truncated spectrum); a pass_store with KB > 0 writes only the band (last pass of
// a transform whose outputs outside it are discarded).
template <int N, int KB> PD_HD bool in_band(int n) { return KB == 0 || n <= KB || n >= N - KB; }

// Of a first pass of radix R (element n = j + r N / R, j < N / R) or a last pass (output n
// likewise), round r lies outside the band for every j (0), below its upper edge (1), above its
// lower edge (2), or either (3: decided per element).
template <int N, int R, int KB> constexpr int band_round(int r) {
    const int lo = r * (N / R), hi = lo + N / R - 1;
    if (KB == 0) return 3;
    if (lo > KB && hi < N - KB) return 0;
    if (hi <= KB) return 1;
    if (lo >= N - KB) return 2;
    return 3;
}
template <int N, int R, int KB> constexpr unsigned zero_mask() {
    unsigned z = 0;
    for (int r = 0; r < R; r++) z |= (band_round<N, R, KB>(r) == 0 ? 1u : 0u) << r;
    return z;
}
// The band class of a round as a type, for load and store functors of truncated transforms.
template <int B> struct Band { static constexpr int value = B; };
template <int I> struct RoundIx { static constexpr int value = I; };
template <int I, int R, class F> PD_HD void for_rounds(F& f) {
    if constexpr (I < R) {
        f(RoundIx<I>{});
        for_rounds<I + 1, R>(f);
    }
}

template <int N, int R, int NS, int S, int L, int LP, int PS = 0, int AS = 0, int KB = 0, class C>
PD_HD void pass_load(const C* s, const C* tw, int w, C* v) {
    using T = real_of<C>;
    constexpr int NR = N / R;
    const int l = item_line<NR, L, AS>(w), j = item_index<NR, L, AS>(w);
    static_assert(KB == 0 || NS == 1, "a band of loads belongs to a first pass");
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int b = band_round<N, R, KB>(r);
        if (KB > 0 && (b == 0 || (b == 3 && !in_band<N, KB>(j + r * NR)))) v[r] = mk(T(0), T(0));
        else v[r] = s[tidx<LP, PS, AS>(j + r * NR, l)];
    }
    if constexpr (NS > 1) {
        const int k = j % NS;
        constexpr int step = N / (NS * R);
        C wt[R];
        twiddles<R>(tw, k * step, wt);
#pragma unroll
        for (int r = 1; r < R; r++) v[r] = twmul<S>(v[r], wt[r]);
    }
    dft<R, S, zero_mask<N, R, KB>()>(v);
}
template <int N, int R, int NS, int L, int LP, int PS = 0, int AS = 0, int KB = 0, class C>
PD_HD void pass_store(C* s, int w, const C* v) {
    const int l = item_line<N / R, L, AS>(w), j = item_index<N / R, L, AS>(w);
    const int k = j % NS;
    const int d = (j / NS) * NS * R + k;
    static_assert(KB == 0 || NS * R == N, "a band of stores belongs to a last pass");
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int b = band_round<N, R, KB>(r);   // of a last pass: d < NS = N / R
        if (KB == 0 || b == 1 || b == 2 || (b == 3 && in_band<N, KB>(d + r * NS))) s[tidx<LP, PS, AS>(d + r * NS, l)] = v[r];
    }
}

// Transforms whose first pass reads global memory and whose last pass writes it
// ("direct" tile transforms).  The L lines of a tile are interleaved in shared
// memory, element n of line l at s[n*L + l] with L = 8: the 8 threads of a
// quarter-warp always own the 8 lines of one butterfly, so every shared access of
// every pass is one contiguous 128-byte row (no bank conflicts, no pad rows), and
// the same 8 threads touch 8 lines x 16 bytes of global memory per element.
// The first pass takes element n of line l from ld(n, l); the last pass hands
// output n of line l to st(n, l, value).  A two-pass length costs one shared-memory
// round trip per element instead of four.
// With KB > 0 (a truncated spectrum) ld and st are called as ld(n, l, Band<B>) and
// st(n, l, value, Band<B>), B the class of the round (band_round): rounds outside the band are
// neither loaded nor stored, and only B = 3 needs a test of n.
template <int N, int R, int S, int L, int KB = 0, int PS = 0, class C, class Ld>
PD_HD void pass_first(C* s, int w, Ld& ld) {
    using T = real_of<C>;
    constexpr int NR = N / R;
    const int l = w % L, j = w / L;
    C v[R];
    auto load = [&](auto ix) {
        constexpr int r = decltype(ix)::value, b = band_round<N, R, KB>(r);
        if constexpr (KB == 0) v[r] = ld(j + r * NR, l);
        else if constexpr (b == 0) v[r] = mk(T(0), T(0));
        else v[r] = ld(j + r * NR, l, Band<b>{});
    };
    for_rounds<0, R>(load);
    dft<R, S, zero_mask<N, R, KB>()>(v);
#pragma unroll
    for (int r = 0; r < R; r++) s[prow<PS>(j * R + r) * L + l] = v[r];
}
template <int N, int R, int S, int L, int KB = 0, int PS = 0, class C, class St>
PD_HD void pass_last(const C* s, const C* tw, int w, St& st) {
    constexpr int NS = N / R;
    C v[R];
    pass_load<N, R, NS, S, L, L, PS>(s, tw, w, v);
    const int l = w % L, j = w / L;
    auto store = [&](auto ix) {
        constexpr int r = decltype(ix)::value, b = band_round<N, R, KB>(r);
        if constexpr (KB == 0) st(j + r * NS, l, v[r]);
        else if constexpr (b != 0) st(j + r * NS, l, v[r], Band<b>{});
    };
    for_rounds<0, R>(store);
}
// Single-pass lengths: global to global, no shared memory.
template <int N, int S, int L, int KF = 0, int KS = 0, class Ld, class St>
PD_HD void pass_only(int l, Ld& ld, St& st) {
    auto get = [&](int n) {
        if constexpr (KF == 0) return ld(n, l);
        else return ld(n, l, Band<3>{});
    };
    using C = decltype(get(0));
    C v[N];
#pragma unroll
    for (int r = 0; r < N; r++) v[r] = get(r);
    dft<N, S>(v);
#pragma unroll
    for (int r = 0; r < N; r++) {
        if constexpr (KS == 0) st(r, l, v[r]);
        else st(r, l, v[r], Band<3>{});
    }
}

// Pad interval (log2) of a tile whose rows (one element of every line) are ROWB bytes, after a
// first pass of radix R0.  Rows of 128 bytes need none.  With shorter rows a wavefront of a store
// of the first pass holds several butterflies' rows, R0 rows apart: for an even R0 in the same
// banks, unless a pad row lies between them.
template <int ROWB, int R0> constexpr int tile_pad() {
    return (ROWB >= 128 || R0 % 2 != 0) ? 0 : (R0 == 8 ? 3 : (R0 == 16 ? 4 : (R0 == 32 ? 5 : (R0 == 4 ? 2 : 0))));
}

// Threads of a tile transform of L lines with the radix plan (R0, R1, R2): one
// butterfly per thread in the pass with the most, 64..512.
template <int N, int R0, int R1, int R2, int L = 8> constexpr int tile_threads_for() {
    constexpr int a = N / R0;
    constexpr int b = R1 ? N / R1 : 0;
    constexpr int c = R2 ? N / R2 : 0;
    constexpr int m = L * (a > b ? (a > c ? a : c) : (b > c ? b : c));
    return m < 64 ? 64 : (m > 512 ? 512 : m);
}

// Radix schedule of the warp-level transforms (one line per warp): radix 8 where
// possible so that a pass has N/8 items, about one per lane.
template <int N> struct WPlan { static constexpr int r0 = 0, r1 = 0, r2 = 0; };
#define PD_WPLAN(N_, A, B, C) \
    template <> struct WPlan<N_> { static constexpr int r0 = A, r1 = B, r2 = C; };
PD_WPLAN(16, 4, 4, 0)
PD_WPLAN(24, 3, 8, 0)
PD_WPLAN(32, 4, 8, 0)
PD_WPLAN(40, 5, 8, 0)
PD_WPLAN(48, 4, 12, 0)
PD_WPLAN(56, 7, 8, 0)
PD_WPLAN(64, 8, 8, 0)
PD_WPLAN(80, 5, 16, 0)
PD_WPLAN(96, 8, 12, 0)
PD_WPLAN(112, 7, 16, 0)
PD_WPLAN(128, 4, 4, 8)
PD_WPLAN(160, 5, 4, 8)
PD_WPLAN(192, 16, 12, 0)
PD_WPLAN(224, 7, 4, 8)
PD_WPLAN(256, 4, 8, 8)
PD_WPLAN(320, 5, 8, 8)
PD_WPLAN(384, 3, 8, 16)
PD_WPLAN(448, 7, 8, 8)
PD_WPLAN(512, 8, 8, 8)
PD_WPLAN(640, 5, 8, 16)
PD_WPLAN(768, 3, 16, 16)
PD_WPLAN(896, 7, 8, 16)
PD_WPLAN(1024, 16, 8, 8)
#undef PD_WPLAN

template <int N> constexpr bool wplan_ok() {
    return WPlan<N>::r0 * (WPlan<N>::r1 ? WPlan<N>::r1 : 1) * (WPlan<N>::r2 ? WPlan<N>::r2 : 1) == N;
}

// Fewer, larger passes for kernels limited by shared-memory bandwidth rather than by registers:
// each pass costs a full read and write of the line.  The two-pass plans of 160 to 448 points
// took the shear step of 160^3 from 0.872 to 0.819 ms (FP32-mixed 0.503 -> 0.452), 224^3 2.27 ->
// 2.02, 320^3 6.6 -> 5.49, 448^3 16.8 -> 13.95 (11.4 -> 7.98); those of 640 to 896 points, which
// in FP32 also let the product step run in registers, 640^3 67.8 -> 63.1 (30.5 -> 22.9), 768^3
// 125.9 -> 117.7 (48.2 -> 39.4), 896^3 181.2 -> 166.0.
template <int N> struct WPlanL : WPlan<N> {};
template <> struct WPlanL<128> { static constexpr int r0 = 16, r1 = 8, r2 = 0; };
template <> struct WPlanL<160> { static constexpr int r0 = 10, r1 = 16, r2 = 0; };
template <> struct WPlanL<224> { static constexpr int r0 = 14, r1 = 16, r2 = 0; };
template <> struct WPlanL<256> { static constexpr int r0 = 16, r1 = 16, r2 = 0; };
template <> struct WPlanL<320> { static constexpr int r0 = 20, r1 = 16, r2 = 0; };
template <> struct WPlanL<384> { static constexpr int r0 = 32, r1 = 12, r2 = 0; };
template <> struct WPlanL<448> { static constexpr int r0 = 28, r1 = 16, r2 = 0; };
template <> struct WPlanL<512> { static constexpr int r0 = 32, r1 = 16, r2 = 0; };
template <> struct WPlanL<640> { static constexpr int r0 = 20, r1 = 32, r2 = 0; };
template <> struct WPlanL<768> { static constexpr int r0 = 24, r1 = 32, r2 = 0; };
template <> struct WPlanL<896> { static constexpr int r0 = 28, r1 = 32, r2 = 0; };
template <> struct WPlanL<1024> { static constexpr int r0 = 32, r1 = 32, r2 = 0; };

// Plan of a backward transform, a pointwise product and a forward transform run
// by one warp (the x pass): backward (r0, r1[, r2]) = WPlanL; with `fused` the
// forward transform runs the reversed plan, so that the last backward pass and
// the first forward pass see the same elements n = j + r * (N / rl) in item j, and
// the last backward pass of one array, the product and the first forward pass run
// in registers, one item per lane (nrl = N / rl items, 16..32 of them).  That is the schedule of
// the lengths whose three arrays do not fit the registers (FP64 from 640 points) and of the
// statistics pass, whose lines shorter than 256 keep separate passes and the same plan both ways;
// elsewhere the product step takes all three arrays (the x pass's `triple`), with the reversed
// plan at every length.
template <int N> struct FusedPlan {
    static constexpr int r0 = WPlanL<N>::r0, r1 = WPlanL<N>::r1, r2 = WPlanL<N>::r2;
    static constexpr int np = r2 ? 3 : 2;
    static constexpr int rl = r2 ? r2 : r1;
    static constexpr int nrl = N / rl;
    static constexpr bool fused = N >= 256 && nrl >= 16 && nrl <= 32;
    static constexpr int f0 = fused ? rl : r0;
    static constexpr int f1 = fused ? (r2 ? r1 : r0) : r1;
    static constexpr int f2 = fused ? (r2 ? r0 : 0) : r2;
};

template <int N> constexpr bool wplanl_ok() {
    return WPlanL<N>::r0 * (WPlanL<N>::r1 ? WPlanL<N>::r1 : 1) * (WPlanL<N>::r2 ? WPlanL<N>::r2 : 1) == N;
}

#if defined(__CUDACC__)
// NA lines transformed in lockstep by one warp (interleaved columns 0..NA-1 for
// AS = 0, else separate arrays AS elements apart): each pass has NA times the
// independent work of a single line, which fills the lanes a radix-16 pass of
// one line leaves idle.
// KL / KS: band of the loads / stores (see in_band).
// W: lanes per line group (32: the whole warp; 32 / W groups of a warp each transform
// their own lines, `lane` being the lane within the group).
template <int N, int R, int NS, int S, int LP, int PS, int NA, int AS = 0, int KL = 0, int KS = 0, int W = 32, class C>
__device__ __forceinline__ void wpass_n(C* s, const C* __restrict__ tw, int lane) {
    if constexpr (NA > 1 && AS > 0 && NS > 1 && N / R == W) {
        // One item per lane and array: the arrays' items of a lane share their twiddles
        // (their products are a sixth of an FP64 radix-16 pass).
        C wt[R], v[NA][R];
        twiddles<R>(tw, (lane % NS) * (N / (NS * R)), wt);
#pragma unroll
        for (int a = 0; a < NA; a++) {
#pragma unroll
            for (int r = 0; r < R; r++) {
                v[a][r] = s[tidx<LP, PS, AS>(lane + r * W, a)];
                if (r > 0) v[a][r] = twmul<S>(v[a][r], wt[r]);
            }
            dft<R, S>(v[a]);
        }
        __syncwarp();
#pragma unroll
        for (int a = 0; a < NA; a++) pass_store<N, R, NS, 1, LP, PS, 0, KS>(s + a * AS, lane, v[a]);
        __syncwarp();
        return;
    }
    constexpr int WORK = (N / R) * NA;
    constexpr int IT = (WORK + W - 1) / W;
    C v[IT][R];
#pragma unroll
    for (int it = 0; it < IT; it++) {
        const int w = lane + it * W;
        if (WORK % W == 0 || w < WORK) pass_load<N, R, NS, S, NA, LP, PS, AS, KL>(s, tw, w, v[it]);
    }
    __syncwarp();
#pragma unroll
    for (int it = 0; it < IT; it++) {
        const int w = lane + it * W;
        if (WORK % W == 0 || w < WORK) pass_store<N, R, NS, NA, LP, PS, AS, KS>(s, w, v[it]);
    }
    __syncwarp();
}

// Passes P0..P1-1 of the radix plan (R0, R1, R2) over NA arrays owned by one
// warp: pass p has radix Rp and NS = the product of the radices before it.  The
// plan's first pass reads the band KL, its last pass writes the band KS.
template <int N, int S, int LP, int PS, int NA, int AS, int R0, int R1, int R2, int P0, int P1,
          int KL = 0, int KS = 0, int W = 32, class C>
__device__ __forceinline__ void wpasses(C* s, const C* __restrict__ tw, int lane) {
    constexpr int NP = R2 ? 3 : (R1 ? 2 : 1);
    if constexpr (P0 <= 0 && 0 < P1) wpass_n<N, R0, 1, S, LP, PS, NA, AS, KL, NP == 1 ? KS : 0, W>(s, tw, lane);
    if constexpr (P0 <= 1 && 1 < P1 && NP > 1) wpass_n<N, R1, R0, S, LP, PS, NA, AS, 0, NP == 2 ? KS : 0, W>(s, tw, lane);
    if constexpr (P0 <= 2 && 2 < P1 && NP > 2) wpass_n<N, R2, R0 * R1, S, LP, PS, NA, AS, 0, KS, W>(s, tw, lane);
}

// In-place pass over a [N][LP] shared tile with NT threads; items w = tid + it*NT.
template <int N, int R, int NS, int S, int L, int LP, int NT, int PS = 0, class C>
__device__ __forceinline__ void pass(C* s, const C* __restrict__ tw, int tid) {
    constexpr int WORK = (N / R) * L;
    constexpr int IT = (WORK + NT - 1) / NT;
    C v[IT][R];
#pragma unroll
    for (int it = 0; it < IT; it++) {
        const int w = tid + it * NT;
        if (WORK % NT == 0 || w < WORK) pass_load<N, R, NS, S, L, LP, PS>(s, tw, w, v[it]);
    }
    __syncthreads();
#pragma unroll
    for (int it = 0; it < IT; it++) {
        const int w = tid + it * NT;
        if (WORK % NT == 0 || w < WORK) pass_store<N, R, NS, L, LP, PS>(s, w, v[it]);
    }
    __syncthreads();
}

// Direct tile transform of L interleaved lines by NT threads (see pass_first) with
// the radix plan (R0, R1, R2), by default Plan<N>.  The caller makes `s` free
// before the call (a barrier after any earlier use); on return other threads may
// still read `s`.  `mid()` runs once per thread after the first pass (the loads
// of the tile are done and the remaining passes are shared-memory work).
struct NoMid {
    __device__ void operator()() const {}
};
// KF, KS: band of the loads and of the stores (0: every element).  PS: one pad row after every
// 2^PS rows (tile_pad).
template <int N, int S, int L, int NT, int R0 = Plan<N>::r0, int R1 = Plan<N>::r1, int R2 = Plan<N>::r2,
          int KF = 0, int KS = 0, int PS = 0, class C, class Ld, class St, class Mid = NoMid>
__device__ __forceinline__ void fft_tile_io(C* s, const C* __restrict__ tw, int tid, Ld& ld, St& st,
                                            const Mid& mid = Mid()) {
    static_assert(R0 * (R1 ? R1 : 1) * (R2 ? R2 : 1) == N, "radix plan does not factor N");
    if constexpr (R1 == 0) {
        mid();
        for (int l = tid; l < L; l += NT) pass_only<N, S, L, KF, KS>(l, ld, st);
    } else {
        constexpr int W0 = (N / R0) * L;
#pragma unroll
        for (int w = tid; w < W0; w += NT) pass_first<N, R0, S, L, KF, PS>(s, w, ld);
        __syncthreads();
        mid();
        if constexpr (R2 != 0) pass<N, R1, R0, S, L, L, NT, PS>(s, tw, tid);   // in place, ends with a barrier
        constexpr int RL = R2 ? R2 : R1;
        constexpr int WL = (N / RL) * L;
#pragma unroll
        for (int w = tid; w < WL; w += NT) pass_last<N, RL, S, L, KS, PS>(s, tw, w, st);
    }
}
#endif

}  // namespace pdfft
