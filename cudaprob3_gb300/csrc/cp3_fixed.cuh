// cp3_fixed.cuh -- the FP64 atmospheric bins in 64-bit fixed point, on the integer pipe.
//
// Why: GB300 retires one FP64 multiply-add per sub-partition and warp in 64 cycles (measured;
// an FP32 one takes one), and the FP64 per-bin kernel was bound by it (89 % of the pipe active).
// Everything after the eigen tables is bounded arithmetic: entries of unitary matrices, sines
// and cosines, probabilities, all at most 1 in magnitude.  As fixed-point numbers with 62
// fraction bits they carry 9 bits more than a double near 1, and a product costs three 32 x 32
// -> 64-bit integer multiply-adds (4.5 cycles each), a quarter of an FP64 one's time.
//
// A value is h 2^-30 + l 2^-62 with both words signed; products keep h h and the two cross
// terms (the dropped l l is below 2^-62).  Sums of products accumulate in 64 bits: by
// Cauchy-Schwarz a dot product of unit vectors with three terms (or two complex ones) keeps
// the cross terms below 2^63 in one accumulator, longer ones use two.
//
// Integer arithmetic but for: a phase's reduction (four FP64 operations), the determinant's of a
// chain's end, the quotients of fx_refine (FP32) and the rates it returns (FP64), the arguments of
// the height sums and sin(x) / x beyond the series (FP64), and the start from double-floats (FP32).
// All of it runs on the host as well, except fx_solve, whose eigen-solver takes paired FP32
// instructions.
#pragma once

#include <cstring>

#include "cp3_device.cuh"

namespace cp3 {

// Table fields (8 bytes each, [class][field][ne_pad], so that a warp reads 256 contiguous bytes
// a field): R_c = U_{c+1}^T U_c row by row as fixed-point word pairs (the rotation from the
// eigenbasis of class c to that of class c + 1; none for the last class), then the phase rates
// of eigenstates 1 and 2 in turns per km as doubles.
constexpr int kFxRates = 9;
constexpr int kFxFields = 11;
// After the classes, once per energy: the electron and muon rows of W U_1 and of W U_0 (three
// real, three complex numbers each; U_c = [u0 u1 u2] of class c, class 0 the air), and the
// coefficients of a bin that crosses no shell.  A table of the air alone holds U_0 in the place
// of the rows of W U_1.
constexpr int kFxV1 = 0, kFxV0 = 9, kFxVac = 18, kFxExtra = 31;

struct fx {
    int h, l;
};
struct cfx {
    fx re, im;
};

CP3_HD fx fx_split(long long v) {
    return fx{(int)(v >> 32) + (int)((unsigned int)v >> 31), (int)v};
}
CP3_HD long long fx_value(fx a) { return (long long)(((unsigned long long)(long long)a.h << 32) + (unsigned long long)(long long)a.l); }
// To one unit, 2^-62: the low word's lowest value has no negative (-l of it is off by 2^-30).
CP3_HD fx fx_neg(fx a) { return fx{-a.h, ~a.l}; }
CP3_HD fx fx_of(int2 v) { return fx{v.x, v.y}; }

// |v| < 2
CP3_HD long long fx_from_double(double v) {
#ifdef __CUDA_ARCH__
    return __double2ll_rn(__dmul_rn(v, 4611686018427387904.0));
#else
    return (long long)llrint(v * 4611686018427387904.0);
#endif
}

CP3_HD long long fx_bits(double v) {
#ifdef __CUDA_ARCH__
    return __double_as_longlong(v);
#else
    long long b;
    std::memcpy(&b, &v, sizeof b);
    return b;
#endif
}
CP3_HD double fx_bits_to_double(long long b) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double(b);
#else
    double v;
    std::memcpy(&v, &b, sizeof v);
    return v;
#endif
}

// A layer's phases are of length 1 to the 2^-56 of their sines and cosines, and the palindrome takes
// a chain twice, so that a probability or a difference of some from 1 leaves [0, 1] by up to about
// M 2^-54 on M shells: -1.1e-15 was met on 59 shells and -2.2e-15 on 128, with theta12 = theta13 = 0,
// where a channel is exactly zero.  A probability as a double, in [0, 1]:
constexpr long long kFxOne = 1LL << 62;
CP3_HD double fx_probability(long long v) {
    if (v <= 0) return 0.0;
    return fx_bits_to_double(fx_bits((double)(v < kFxOne ? v : kFxOne)) - (62LL << 52));
}

// An averaged one: the end of the interval within that rounding (2^-47) outside it, else what it is.
// Weights that are no distribution, and the jump of the sinc series (fx_sinc) where two states are
// nearly degenerate, take it out.
CP3_HD double fx_to_double(long long v) {
    constexpr long long window = 1LL << 15;
    if (v <= 0 && v > -window) return 0.0;
    if (v > kFxOne && v < kFxOne + window) return 1.0;
    return fx_bits_to_double(fx_bits((double)v) - (62LL << 52));
}

// Accumulators: fxacc for at most three products of unit-vector entries (two of complex ones),
// fxacc2, whose cross terms have an accumulator each, for up to three complex products.
struct fxacc {
    long long hh = 0, x = 0;
};
struct fxacc2 {
    long long hh = 0, x = 0, y = 0;
};
// s + a b and a b, 32 x 32 -> 64 bits.  Stated as the instruction they are: from the products of
// widened operands the compiler made a fifth more of them (59 shells,
// 2000 x 2000: 1.48 ms, and 1.15 so; 1.12 with the sums' halves joined by the high word alone).
CP3_HD void fx_mad(long long& s, int a, int b) {
#ifdef __CUDA_ARCH__
    asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(s) : "r"(a), "r"(b));
#else
    s += (long long)a * b;
#endif
}
CP3_HD long long fx_mul(int a, int b) {
#ifdef __CUDA_ARCH__
    long long s;
    asm("mul.wide.s32 %0, %1, %2;" : "=l"(s) : "r"(a), "r"(b));
    return s;
#else
    return (long long)a * b;
#endif
}
CP3_HD void fx_mac(fxacc& s, fx a, fx b) {
    fx_mad(s.hh, a.h, b.h);
    fx_mad(s.x, a.h, b.l);
    fx_mad(s.x, a.l, b.h);
}
CP3_HD void fx_mac(fxacc2& s, fx a, fx b) {
    fx_mad(s.hh, a.h, b.h);
    fx_mad(s.x, a.h, b.l);
    fx_mad(s.y, a.l, b.h);
}
CP3_HD long long fx_sum(const fxacc& s) { return (s.hh + (s.x >> 32)) * 4; }  // to 2^-60
CP3_HD long long fx_sum(const fxacc2& s) { return (s.hh + (s.x >> 32) + (s.y >> 32)) * 4; }
template <class Acc>
CP3_HD fx fx_res(const Acc& s) {
    return fx_split(fx_sum(s));
}

// a b for |a| = 1
CP3_HD cfx fx_cmul(cfx a, cfx b) {
    const fx n = fx_neg(a.im);
    fxacc r, i;
    fx_mac(r, a.re, b.re);
    fx_mac(r, n, b.im);
    fx_mac(i, a.re, b.im);
    fx_mac(i, a.im, b.re);
    return cfx{fx_res(r), fx_res(i)};
}

// ---- sine and cosine --------------------------------------------------------------------
// cos and sin of 2 pi k / 512, 62 fraction bits, evaluated by the compiler: the Taylor series
// of the angle's distance to the nearest axis, at most pi / 4, in 62-bit fixed point (a few
// units of 2^-62).
constexpr int kTrigBits = 9, kTrigSize = 1 << kTrigBits;

struct TrigTable {
    long long cs[kTrigSize][2];
};

constexpr long long trig_mul(long long a, long long b) { return (long long)(((__int128)a * b + ((__int128)1 << 61)) >> 62); }

constexpr TrigTable make_trig_table() {
    TrigTable t{};
    const long long one = 1LL << 62;
    const __int128 pi60 = 3622009729038561421LL;  // pi 2^60
    for (int k = 0; k <= kTrigSize / 8; k++) {
        const long long x = (long long)((pi60 * k * 4 + kTrigSize / 4) / (kTrigSize / 2));  // 2 pi k / 512
        const long long x2 = trig_mul(x, x);
        long long s = 0, c = 0;  // Horner: 1 - x^2/(n (n-1)) (1 - ...)
        for (int n = 24; n >= 2; n -= 2) {
            c = one - trig_mul(x2, (n == 24 ? one : c)) / (n * (n - 1));
            s = one - trig_mul(x2, (n == 24 ? one : s)) / (n * (n + 1));
        }
        s = trig_mul(x, s);
        if (k == 0) {
            c = one;
            s = 0;
        }
        const int q = kTrigSize / 4;
        // the eight octants
        t.cs[k][0] = c, t.cs[k][1] = s;
        t.cs[q - k][0] = s, t.cs[q - k][1] = c;
        t.cs[q + k][0] = -s, t.cs[q + k][1] = c;
        t.cs[2 * q - k][0] = -c, t.cs[2 * q - k][1] = s;
        t.cs[2 * q + k][0] = -c, t.cs[2 * q + k][1] = -s;
        t.cs[3 * q - k][0] = -s, t.cs[3 * q - k][1] = -c;
        t.cs[3 * q + k][0] = s, t.cs[3 * q + k][1] = -c;
        t.cs[(4 * q - k) % kTrigSize][0] = c, t.cs[(4 * q - k) % kTrigSize][1] = -s;
    }
    t.cs[0][1] = 0;
    return t;
}

// A phase of t = w L turns: table index (t in 512ths, any integer multiple of 512 away) and the
// remaining angle in radians, 58 fraction bits, |x| <= pi / 512.
struct FxAngle {
    int k;
    long long x;
};

// w L is rounded to a multiple of 1/512 by adding 1.5 2^43 (whose last place that is); the FMA
// leaves the remainder of the exact product with one rounding, 2^-63, and another FMA takes it
// to radians in the last places of 1.5 2^-6.  `bad` collects the exponents: bits above 19 come
// up where w L is not finite or beyond 2^42 turns, and the caller takes the FP64 path then.
CP3_HD FxAngle fx_angle(double w, double L, unsigned int& bad) {
    constexpr double kRound = 13194139533312.0;  // 1.5 2^43
    constexpr double kPlace = 0.0234375;         // 1.5 2^-6
    const double q = fma(w, L, kRound);
    const double n = q - kRound;
    const double r = fma(w, L, -n);
    const double u = fma(r, 6.283185307179586477, kPlace);
    const long long qb = fx_bits(q), ub = fx_bits(u);
    bad |= (unsigned int)(qb >> 32) ^ 0x42A00000u;
    bad |= (unsigned int)(ub >> 32) ^ 0x3F900000u;
    return FxAngle{(int)qb, ub - 0x3F98000000000000LL};
}

// cos and sin of an angle: the table's entry T rotated by the remaining x, with
// sin x = x (1 - p), p = x^2/6 (1 - x^2/20), and cos x - 1 = -x^2/2 (1 - s),
// s = x^2/12 (1 - x^2/30); |x| <= 0.0062, so p and s need one word.  x, sin x and cos x - 1 are
// held times 2^7.  Error about 2^-56 (an FP64 sincos rounds at 2^-54).
CP3_HD void fx_sincos(FxAngle a, const longlong2* trig, fx& c, fx& s) {
    const longlong2 T = trig[a.k & (kTrigSize - 1)];
    const fx tc = fx_split(T.x), ts = fx_split(T.y), nts = fx_neg(ts);
    const long long X = a.x << 11;
    const fx x = fx_split(X);
    const long long w = fx_mul(x.h, x.h) * 4 + (fx_mul(x.h, x.l) >> 29);  // x^2 2^14
    const int w31 = (int)(w >> 31);                                        // 31 fraction bits
    const int d = (int)(fx_mul(w31, 8738) >> 32);                          // (4/3) 2^30 x^2/20
    const int p48 = (int)(fx_mul(w31, 1431655765 - d) >> 30);              // p 2^48
    const unsigned int s48 = (unsigned int)(((unsigned long long)(unsigned int)w31 * (2863311531u - (unsigned int)(d + (d >> 2)))) >> 32);
    long long xp = fx_mul(x.l, p48) >> 32;
    fx_mad(xp, x.h, p48);
    const fx sn = fx_split(X - (xp >> 16));
    const fx cm = fx_split((fx_mul(w31, (int)s48) >> 25) - (w >> 8));
    fxacc ac, as;
    fx_mac(ac, tc, cm);
    fx_mac(ac, nts, sn);
    fx_mac(as, ts, cm);
    fx_mac(as, tc, sn);
    c = fx_split(T.x + ((ac.hh + (ac.x >> 32)) >> 5));
    s = fx_split(T.y + ((as.hh + (as.x >> 32)) >> 5));
}

// e^{-i phi} of one phase; k and x add up to the determinant's phase.
CP3_HD cfx fx_unit(FxAngle a, const longlong2* trig) {
    cfx e;
    fx_sincos(a, trig, e.re, e.im);
    e.im = fx_neg(e.im);
    return e;
}

// ---- a bin ------------------------------------------------------------------------------
// One energy column of the table.
struct FxColumn {
    const int2* tab;   // at this energy: field f of class c at tab[c * cls_stride + f * stride]
    const int2* ext;   // extra field f at ext[f * stride]
    size_t stride, cls_stride;
    CP3_HD int2 load(const int2* p) const {
#ifdef __CUDA_ARCH__
        return __ldca(p);  // (written while this grid is already there: launch_early)
#else
        return *p;
#endif
    }
    CP3_HD fx rot(int c, int f) const { return fx_of(load(tab + c * cls_stride + f * stride)); }
    CP3_HD fx extra(int f) const { return fx_of(load(ext + f * stride)); }
    CP3_HD double rate(int c, int k) const {
        const int2 v = load(tab + c * cls_stride + (kFxRates + k) * stride);
        return fx_bits_to_double((long long)(((unsigned long long)(unsigned int)v.y << 32) | (unsigned int)v.x));
    }
};

CP3_HD void fx_load_rotation(const FxColumn& t, int c, fx R[9]) {
#pragma unroll
    for (int f = 0; f < 9; f++) R[f] = t.rot(c, f);
}

// v <- R v
CP3_HD void fx_rotate(const fx R[9], cfx v[3]) {
    cfx o[3];
#pragma unroll
    for (int i = 0; i < 3; i++) {
        fxacc r, m;
#pragma unroll
        for (int k = 0; k < 3; k++) {
            fx_mac(r, R[i * 3 + k], v[k].re);
            fx_mac(m, R[i * 3 + k], v[k].im);
        }
        o[i] = cfx{fx_res(r), fx_res(m)};
    }
#pragma unroll
    for (int i = 0; i < 3; i++) v[i] = o[i];
}

// sum_k a_k b_k over three complex products
CP3_HD cfx fx_cdot(cfx a0, cfx b0, cfx a1, cfx b1, cfx a2, cfx b2) {
    fxacc2 r, m;
    fx_mac(r, a0.re, b0.re), fx_mac(r, fx_neg(a0.im), b0.im), fx_mac(m, a0.re, b0.im), fx_mac(m, a0.im, b0.re);
    fx_mac(r, a1.re, b1.re), fx_mac(r, fx_neg(a1.im), b1.im), fx_mac(m, a1.re, b1.im), fx_mac(m, a1.im, b1.re);
    fx_mac(r, a2.re, b2.re), fx_mac(r, fx_neg(a2.im), b2.im), fx_mac(m, a2.re, b2.im), fx_mac(m, a2.im, b2.re);
    return cfx{fx_res(r), fx_res(m)};
}

// conj(a x b)_i for entries j, k = i + 1, i + 2
CP3_HD cfx fx_cross(cfx aj, cfx ak, cfx bj, cfx bk) {
    fxacc2 r, m;
    fx_mac(r, aj.re, bk.re), fx_mac(r, fx_neg(aj.im), bk.im), fx_mac(r, fx_neg(ak.re), bj.re), fx_mac(r, ak.im, bj.im);
    const fx njr = fx_neg(aj.re), nji = fx_neg(aj.im);
    fx_mac(m, njr, bk.im), fx_mac(m, nji, bk.re), fx_mac(m, ak.re, bj.im), fx_mac(m, ak.im, bj.re);
    return cfx{fx_res(r), fx_res(m)};
}

CP3_HD long long fx_norm(cfx a) {
    fxacc s;
    fx_mac(s, a.re, a.re);
    fx_mac(s, a.im, a.im);
    return fx_sum(s);
}

// y <- D y for the phases e of one layer
CP3_HD void fx_phase(const cfx e[2], cfx y[3]) {
    y[1] = fx_cmul(e[0], y[1]);
    y[2] = fx_cmul(e[1], y[2]);
}

// The sum of the layers' phases: e^{-i (sum)} is the determinant of their product.
struct FxDet {
    int k = 0;
    long long x = 0;
};

// The two phases of one layer; `det` collects them where given.
CP3_HD void fx_layer(const double rate[2], double L, const longlong2* trig, cfx e[2], unsigned int& bad,
                     FxDet* det = nullptr) {
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const FxAngle a = fx_angle(rate[k], L, bad);
        if (det) {
            det->k += a.k;
            det->x += a.x;
        }
        e[k] = fx_unit(a, trig);
    }
}

// The third column of a unitary matrix from two: det conj(y0 x y1).
CP3_HD void fx_third_column(const FxDet& s, const longlong2* trig, cfx y[3][3]) {
    // the phase is 2 pi k / 512 + x; x is brought back below pi / 512
    const double x = (double)s.x * 3.469446951953614189e-18;  // 2^-58
    const double m = rint(x * 81.48733086305041);             // 512 / (2 pi)
    FxAngle d;
    d.k = s.k + (int)m;
    d.x = s.x - (long long)(int)m * 3537118876014220LL;  // (2 pi / 512) 2^58
    const cfx det = fx_unit(d, trig);
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const int j = (i + 1) % 3, k = (i + 2) % 3;
        y[2][i] = fx_cmul(det, fx_cross(y[0][j], y[0][k], y[1][j], y[1][k]));
    }
}

// k <- Y^T D Y k for Y with columns y[0..2]
CP3_HD void fx_palindrome(const cfx y[3][3], const cfx e[2], cfx k[3]) {
    cfx m[3];
#pragma unroll
    for (int i = 0; i < 3; i++) m[i] = fx_cdot(y[0][i], k[0], y[1][i], k[1], y[2][i], k[2]);
    fx_phase(e, m);
#pragma unroll
    for (int i = 0; i < 3; i++) k[i] = fx_cdot(y[i][0], m[0], y[i][1], m[1], y[i][2], m[2]);
}

// The four probabilities of a single layer from its coefficients (fx_coefficients) and phases:
// P = P0 + sum_k d_k cos D_k for the two survivals, and for the pair the same plus or minus
// J (sin D10 - sin D20 + sin D21).
CP3_HD void fx_one_layer(const fx v[13], const cfx e[2], long long P[4]) {
    fxacc a, b;
    fx_mac(a, e[0].re, e[1].re), fx_mac(a, e[0].im, e[1].im);          // cos D21
    fx_mac(b, e[0].im, e[1].re), fx_mac(b, fx_neg(e[0].re), e[1].im);  // sin D21 (e.im = -sin)
    const fx c3 = fx_res(a);
    const long long sines = (fx_value(e[1].im) >> 1) - (fx_value(e[0].im) >> 1) + (fx_sum(b) >> 1);
    long long r[3];
#pragma unroll
    for (int q = 0; q < 3; q++) {
        fxacc2 s;
        fx_mac(s, v[4 * q + 1], e[0].re);
        fx_mac(s, v[4 * q + 2], e[1].re);
        fx_mac(s, v[4 * q + 3], c3);
        r[q] = fx_value(v[4 * q]) + fx_sum(s);
    }
    fxacc j;
    fx_mac(j, v[12], fx_split(sines));
    const long long jt = fx_sum(j);
    P[0] = r[0];
    P[1] = r[2] + jt;
    P[2] = r[2] - jt;
    P[3] = r[1];
}

// The columns of Y (see fx_bin) for M > 1 table layers; layer(l, e, &det) forms the phases of
// layer l.
template <class Layer>
CP3_HD void fx_columns(const FxColumn& t, int M, Layer layer, const longlong2* trig, cfx y[3][3]) {
    FxDet det;
    cfx e[2];
    layer(1, e, &det);
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const fx a = t.rot(1, 3 * i), b = t.rot(1, 3 * i + 1);
        fxacc r, m;
        fx_mac(r, b, e[0].re);
        fx_mac(m, b, e[0].im);
        y[0][i] = cfx{a, fx{0, 0}};
        y[1][i] = cfx{fx_res(r), fx_res(m)};
    }
#pragma unroll 1
    for (int l = 2; l < M; l++) {
        fx R[9];
        fx_load_rotation(t, l, R);
        layer(l, e, &det);
#pragma unroll
        for (int j = 0; j < 2; j++) {
            fx_phase(e, y[j]);
            fx_rotate(R, y[j]);
        }
    }
    fx_third_column(det, trig, y);
}

// (W U_1) k, rows e and mu: the table's flavour rows of class 1 on a vector in its eigenbasis.
CP3_HD void fx_rows_of(const FxColumn& t, const cfx k[3], cfx& ae, cfx& am) {
    fxacc r, m;
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const fx v = t.extra(kFxV1 + i);
        fx_mac(r, v, k[i].re);
        fx_mac(m, v, k[i].im);
    }
    ae = cfx{fx_res(r), fx_res(m)};
    am = fx_cdot(cfx{t.extra(kFxV1 + 3), t.extra(kFxV1 + 6)}, k[0], cfx{t.extra(kFxV1 + 4), t.extra(kFxV1 + 7)}, k[1],
                 cfx{t.extra(kFxV1 + 5), t.extra(kFxV1 + 8)}, k[2]);
}

// The four probabilities e->e, e->mu, mu->e, mu->mu (62 fraction bits) of one bin over M + 1
// segments (lengths len[0..M] in km; segment l is class l); the other five follow from
// unitarity.  Returns false where a phase left the reduction's range.
//
// With U_l the eigenvectors of layer l (columns, det = 1), D_l = diag(1, e1, e2) its phases and
// R_l = U_{l+1}^T U_l, the amplitude W (S_1..S_{M-1}) S_M (S_{M-1}..S_1) S_0 W^+ of
// S_l = U_l D_l U_l^T is
//   A = (W U_1) Y^T D_M Y R_0 D_0 (W U_0)^+,   Y = R_{M-1} D_{M-1} ... R_1 D_1,
// so a layer costs two complex multiplications and one real rotation per column of Y.  Y is
// unitary with determinant e^{-i sum of the phases}: two of its columns are carried, 52
// multiplications a layer (two rank-1 updates of three columns took 96), and the third is
// det Y conj(y0 x y1) at the end.  Only the columns e and mu of A, and of these the rows e and
// mu, are formed.
CP3_HD bool fx_bin(const FxColumn& t, const double* len, int M, const longlong2* trig, long long P[4]) {
    unsigned int bad = 0;
    cfx e[2];
    auto layer = [&](int l, cfx* f, FxDet* det) {
        const double rate[2] = {t.rate(l, 0), t.rate(l, 1)};
        fx_layer(rate, len[l], trig, f, bad, det);
    };
    if (M == 0) {
        layer(0, e, nullptr);
        fx v[13];
#pragma unroll
        for (int f = 0; f < 13; f++) v[f] = t.extra(kFxVac + f);
        fx_one_layer(v, e, P);
        return (bad >> 20) == 0;
    }
    cfx y[3][3];
    if (M > 1) fx_columns(t, M, layer, trig, y);
    cfx e0[2];
    layer(0, e0, nullptr);
    layer(M, e, nullptr);
    fx R0[9];
    fx_load_rotation(t, 0, R0);
#pragma unroll 1
    for (int j = 0; j < 2; j++) {  // initial flavours e, mu
        cfx k[3];
        // D_0 (W U_0)^+ column j
#pragma unroll
        for (int i = 0; i < 3; i++)
            k[i] = j == 0 ? cfx{t.extra(kFxV0 + i), fx{0, 0}}
                          : cfx{t.extra(kFxV0 + 3 + i), fx_neg(t.extra(kFxV0 + 6 + i))};
        fx_phase(e0, k);
        fx_rotate(R0, k);
        if (M > 1)
            fx_palindrome(y, e, k);
        else
            fx_phase(e, k);
        cfx ae, am;
        fx_rows_of(t, k, ae, am);
        P[2 * j] = fx_norm(ae);
        P[2 * j + 1] = fx_norm(am);
    }
    return (bad >> 20) == 0;
}

// All nine from the four: channel a*3+b at out[ch * plane].
CP3_HD void fx_store(const long long P[4], double* __restrict__ out, size_t plane) {
    const long long one = 1LL << 62;
    const long long et = one - P[0] - P[1], mt = one - P[2] - P[3];
    out[0] = fx_probability(P[0]);
    out[plane] = fx_probability(P[1]);
    out[2 * plane] = fx_probability(et);
    out[3 * plane] = fx_probability(P[2]);
    out[4 * plane] = fx_probability(P[3]);
    out[5 * plane] = fx_probability(mt);
    out[6 * plane] = fx_probability(one - P[0] - P[2]);
    out[7 * plane] = fx_probability(one - P[1] - P[3]);
    out[8 * plane] = fx_probability(one - et - mt);
}

// ---- eigen-systems ----------------------------------------------------------------------
// One layer: U as nine fixed-point numbers (columns u0, u1, u2, det = 1) and the phase rates
// 2.534 (m_k - m_0) / (2 pi E), k = 1, 2, in turns per km.  NaN rates mark a layer whose bins
// take the FP64 path.
struct FxClass {
    fx U[3][3];  // [component][eigenstate]
    double rate[2];
};

constexpr double kFxTurns = 0.40329862579486275;  // 2.534 / (2 pi)

// v / 2^(kexp - 1023), |v| below that power of two, from the bits (truncated at 2^-62); kexp is
// a biased double exponent.
CP3_HD long long fx_scaled(double v, int kexp) {
    const long long b = fx_bits(v);
    const int e = (int)((b >> 52) & 0x7ff);
    const long long m = (long long)(((unsigned long long)b & 0xfffffffffffffull) | 0x10000000000000ull) << 10;
    const int sh = kexp - e;
    const long long r = e == 0 || sh > 62 ? 0 : m >> sh;
    return b < 0 ? -r : r;
}
CP3_HD int fx_exponent(double v) { return (int)((fx_bits(v) >> 52) & 0x7ff); }

// u0 = u1 x u2
CP3_HD void fx_third(fx U[3][3]) {
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const int j = (i + 1) % 3, k = (i + 2) % 3;
        fxacc s;
        fx_mac(s, U[j][1], U[k][2]);
        fx_mac(s, fx_neg(U[k][1]), U[j][2]);
        U[i][0] = fx_res(s);
    }
}

// C = U^T U - 1 (upper triangle); false unless within 2^-31 of orthonormal
CP3_HD bool fx_overlap(const fx U[3][3], int C[6]) {
    bool ok = true;
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = i; j < 3; j++) {
            fxacc s;
#pragma unroll
            for (int k = 0; k < 3; k++) fx_mac(s, U[k][i], U[k][j]);
            const long long v = fx_sum(s) - (i == j ? 1LL << 62 : 0);
            C[sidx(i, j)] = (int)v;
            ok = ok && v == (int)v;
        }
    return ok;
}

// U <- U + U X, X small, in units of 2^-62
CP3_HD void fx_adjust(fx U[3][3], const int X[3][3]) {
#pragma unroll
    for (int i = 0; i < 3; i++) {
        fx r[3];
#pragma unroll
        for (int j = 0; j < 3; j++) {
            long long s = 0;
#pragma unroll
            for (int k = 0; k < 3; k++) fx_mad(s, U[i][k].h, X[k][j]);
            r[j] = fx_split(fx_value(U[i][j]) + (s >> 30));
        }
#pragma unroll
        for (int j = 0; j < 3; j++) U[i][j] = r[j];
    }
}

// From a nearly exact U to the eigen-system of H0 + V e0 e0^T in the last places of the
// fixed-point numbers.  With M = U^T H U (H scaled below 1 by a power of two) and
// C = U^T U - 1, the eigenvalues are M_ii - C_ii M_ii and the vectors U (1 + K - C / 2) with
// K_ij = (M_ij - C_ij (M_ii + M_jj) / 2) / (m_j - m_i): first-order perturbation theory on top
// of a start that is off by 1e-12 at most, so what is left is below 2^-62 (tested: K and C
// within 2^-32 and 2^-31).  The phase rates come from the refined eigenvalues.
//   C / 2 is the Newton-Schulz step to the nearest orthonormal U.  It is not optional: a layer
// is U D U^T, near 1 whatever the rotation U where its phases are small, but only if
// U U^T = 1.  With U orthonormal to FP64 rounding alone that rounding entered every layer
// (59 shells at 100 GeV: 1.4e-14 instead of 1e-15).
//   The same FP64 work -- the cubic's roots by the trigonometric formula, projectors, their
// vectors -- took about 400 FP64 instructions (64 cycles each); this takes about 220 integer
// multiply-adds (4.5 cycles) and 15 FP64 instructions.
CP3_HD bool fx_refine(const OscParams* __restrict__ p, double E, double rE, double rho, FxClass& o) {
    const double V = p->anti ? -(kTwoRtTwoGf * E * rho) : kTwoRtTwoGf * E * rho;
    int kexp = fx_exponent(V);
    const int k1 = fx_exponent(p->dm[3]), k2 = fx_exponent(p->dm[6]);
    kexp = kexp > k1 ? kexp : k1;
    kexp = (kexp > k2 ? kexp : k2) + 3;  // |V| + max |mu| < 2^(kexp - 1023) / 2
    fx H[6];
#pragma unroll
    for (int q = 0; q < 6; q++) {
        const long long h = fx_scaled(p->h0[q], kexp);
        H[q] = fx_split(q == 0 ? h + fx_scaled(V, kexp) : h);
    }
    int C[6];
    bool ok = fx_overlap(o.U, C);
    long long M[6];
#pragma unroll
    for (int j = 0; j < 3; j++) {
        fx g[3];
#pragma unroll
        for (int i = 0; i < 3; i++) {
            fxacc s;
#pragma unroll
            for (int k = 0; k < 3; k++) fx_mac(s, H[sidx(i, k)], o.U[k][j]);
            g[i] = fx_res(s);
        }
#pragma unroll
        for (int i = 0; i <= j; i++) {
            fxacc s;
#pragma unroll
            for (int k = 0; k < 3; k++) fx_mac(s, o.U[k][i], g[k]);
            M[sidx(i, j)] = fx_sum(s);
        }
    }
    long long m[3];
    int mh[3];
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const long long d = M[sidx(i, i)];
        mh[i] = (int)(d >> 32);  // 30 fraction bits
        m[i] = d - (fx_mul(mh[i], C[sidx(i, i)]) >> 30);
    }
    int X[3][3];
#pragma unroll
    for (int i = 0; i < 3; i++) {
        X[i][i] = -(C[sidx(i, i)] >> 1);
#pragma unroll
        for (int j = i + 1; j < 3; j++) {
            const int c = C[sidx(i, j)];
            const long long off = M[sidx(i, j)] - (fx_mul((mh[i] + mh[j]) >> 1, c) >> 30);
            // (float of the difference of the leading words is enough: K is a correction)
            const float k = (float)off / ((float)(m[j] - m[i]) * 2.168404344971009e-19f);  // 2^-62
            ok = ok && fabsf(k) < 1073741824.0f;
            const int ki = ok ? (int)k : 0;
            X[i][j] = ki - (c >> 1);
            X[j][i] = -ki - (c >> 1);
        }
    }
    fx_adjust(o.U, X);
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const long long d = m[k + 1] - m[0];
        // the difference in eV^2
        const double dm = d == 0 ? 0.0 : fx_bits_to_double(fx_bits((double)d) + ((long long)(kexp - 1023 - 62) << 52));
        o.rate[k] = ok ? dm * kFxTurns * rE : fx_bits_to_double(0x7ff8000000000000LL);
    }
    return ok;
}

// The layer from FP64 vectors and masses (rotated_layer_f64): where the fast solver declines.  Of two
// nearly equal levels (below 1e-6 of the spread) the vectors, each from a projector of its own, are
// further from orthogonal than one symmetric step mends, and it is taken again.  (Their bins took
// the FP64 path: PREM-4, 200 x 160 with dm23sq = 1e-10 eV^2 177 us a call and 1.2e-9 from the
// reference's formulas, so 47 us and 1e-10.)
CP3_HD bool fx_entry_ok(double v) { return (unsigned int)((fx_bits(v) >> 32) & 0x7fffffff) <= 0x3FF00010u; }

CP3_HD void fx_class_f64(double u[2][3], const double dmv[3], double E, FxClass& o) {
    int C[6], X[3][3];
    bool ok = false;
#pragma unroll 1
    for (int again = 0; again < 3 && !ok; again++) {
        if (again) orthonormalize_pair(u[0], u[1]);
        ok = true;
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int k = 0; k < 2; k++) {
                ok = ok && fx_entry_ok(u[k][i]);
                o.U[i][k + 1] = fx_split(fx_from_double(u[k][i]));
            }
        fx_third(o.U);
        ok = ok && fx_overlap(o.U, C);
    }
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) X[i][j] = -(C[sidx(i, j)] >> 1);
    fx_adjust(o.U, X);
#pragma unroll
    for (int k = 0; k < 2; k++)
        o.rate[k] = ok ? (dmv[k + 1] - dmv[0]) * kFxTurns / E : fx_bits_to_double(0x7ff8000000000000LL);
}

CP3_HD unsigned int fx_float_bits(float x) {
#ifdef __CUDA_ARCH__
    return __float_as_uint(x);
#else
    unsigned int b;
    std::memcpy(&b, &x, sizeof b);
    return b;
#endif
}
CP3_HD float fx_bits_to_float(unsigned int b) {
#ifdef __CUDA_ARCH__
    return __uint_as_float(b);
#else
    float x;
    std::memcpy(&x, &b, sizeof x);
    return x;
#endif
}

// x as a float pair, from its bits (conversions between double and float take the FP64 pipe);
// false outside 2^-60..2^61 and for what is no number.
CP3_HD bool fx_float_pair(double x, df& o) {
    const long long b = fx_bits(x);
    const int e = fx_exponent(x);
    if ((unsigned long long)b << 1 == 0) {
        o = df{0.0f, 0.0f};
        return true;
    }
    if (e < 1023 - 60 || e > 1023 + 60) return false;
    const unsigned int sign = b < 0 ? 0x80000000u : 0u;
    const float hi = fx_bits_to_float(sign | ((unsigned int)(e - 896) << 23) | ((unsigned int)(b >> 29) & 0x7fffffu));
    const float lo = (float)(unsigned int)(b & 0x1fffffff) * fx_bits_to_float(sign | ((unsigned int)(e - 948) << 23));
    o = df_fast2sum(hi, lo);
    return true;
}
CP3_HD double fx_to_f64(float x) {  // normal or zero (zero: 1e-38)
    const unsigned int b = fx_float_bits(x);
    return fx_bits_to_double((long long)((unsigned long long)((b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + 0x38000000u)) << 32 |
                                         (unsigned int)(b << 29)));
}
CP3_HD fx fx_from_pair(float hi, float lo) {  // |hi + lo| <= 1
#ifdef __CUDA_ARCH__
    const int i = __float2int_rn(hi * 1073741824.0f);
#else
    const int i = (int)rintf(hi * 1073741824.0f);
#endif
    const float rest = fmaf(-(float)i, 9.31322574615478515625e-10f, hi) + lo;  // 2^-30
#ifdef __CUDA_ARCH__
    const long long r = __float2ll_rn(rest * 4611686018427387904.0f);
#else
    const long long r = (long long)rintf(rest * 4611686018427387904.0f);
#endif
    return fx_split((long long)((unsigned long long)(long long)i << 32) + r);
}

// 1 / E, rounded once but for a last-place error of the correction
CP3_HD double fx_reciprocal(double E, df Ed) {
    const df r = df_recip(Ed);
    const double r0 = fx_to_f64(r.hi) + fx_to_f64(r.lo);
    return fma(fma(-E, r0, 1.0), r0, r0);
}

#ifdef __CUDACC__
static __device__ __noinline__ void fx_solve_f64(const OscParams* __restrict__ p, double E, double rho, FxClass* o) {
    double u[2][3], dmv[3];
    rotated_layer_f64(p, E, rho, u, dmv);
    fx_class_f64(u, dmv, E, *o);
}

// The layer of one (energy, electron density): double-float roots and vectors on the FP32 pipe
// (rotated_eigen_mixed_try, 1e-14), refined in fixed point; the FP64 formulas where two levels
// nearly meet or the vectors' formula has no content.
__device__ __forceinline__ void fx_solve(const OscParams* __restrict__ p, double E, double rho, FxClass& o) {
    df Ed, rd;
    df2 v[3];
    float none[2][3], om[2][2];
    bool ok = fx_float_pair(E, Ed) && fx_float_pair(rho, rd) &&
              rotated_eigen_mixed_try<true>(p, Ed, rd, none, om, v);
    if (ok) {
#pragma unroll
        for (int i = 0; i < 3; i++) {
            o.U[i][1] = fx_from_pair(v[i].hi.x, v[i].lo.x);
            o.U[i][2] = fx_from_pair(v[i].hi.y, v[i].lo.y);
        }
        fx_third(o.U);
        ok = fx_refine(p, E, fx_reciprocal(E, Ed), rho, o);
    }
    if (!ok) {
        FxClass t;  // (its own storage: taking o's address would put it in local memory)
        fx_solve_f64(p, E, rho, &t);
        o = t;
    }
}
#endif

// R = B^T A
CP3_HD void fx_rotation(const fx B[3][3], const fx A[3][3], fx R[3][3]) {
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) {
            fxacc s;
#pragma unroll
            for (int k = 0; k < 3; k++) fx_mac(s, B[k][i], A[k][j]);
            R[i][j] = fx_res(s);
        }
}

// The electron and muon rows of W U: U_e (real), and c u_1 + s e^{i d} u_2 as three real and
// three imaginary parts; w = {c23, s23, cos d, sin d}.
CP3_HD void fx_rows(const fx U[3][3], const double* w, fx row[9]) {
    const fx c = fx_split(fx_from_double(w[0])), sr = fx_split(fx_from_double(w[1] * w[2])),
             si = fx_split(fx_from_double(w[1] * w[3]));
#pragma unroll
    for (int k = 0; k < 3; k++) {
        fxacc r, m;
        fx_mac(r, c, U[1][k]);
        fx_mac(r, sr, U[2][k]);
        fx_mac(m, si, U[2][k]);
        row[k] = U[0][k];
        row[3 + k] = fx_res(r);
        row[6 + k] = fx_res(m);
    }
}

// The coefficients of a single layer (a bin that crosses no shell, a beam) from its flavour
// rows: the expansion of layer_coefficients64 in cos D_jk itself.  For e->e, mu->mu and the mean
// of e->mu and mu->e a constant and the factors of cos D10, cos D20, cos D21; then 2 J of the
// sines, doubled.
CP3_HD void fx_coefficients(const fx row[9], fx v[13]) {
    fx m[2][3];
    long long mv[2][3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        fxacc a, b;
        fx_mac(a, row[k], row[k]);
        fx_mac(b, row[3 + k], row[3 + k]);
        fx_mac(b, row[6 + k], row[6 + k]);
        mv[0][k] = fx_sum(a);
        mv[1][k] = fx_sum(b);
        m[0][k] = fx_split(mv[0][k]);
        m[1][k] = fx_split(mv[1][k]);
    }
    auto mul = [](fx a, fx b) {
        fxacc s;
        fx_mac(s, a, b);
        return fx_sum(s);
    };
    auto put = [&](int q, long long c0, long long a, long long b, long long c) {
        v[4 * q] = fx_split(c0 - a - b - c);
        v[4 * q + 1] = fx_split(a);
        v[4 * q + 2] = fx_split(b);
        v[4 * q + 3] = fx_split(c);
    };
#pragma unroll
    for (int q = 0; q < 2; q++)
        put(q, 1LL << 62, 2 * mul(m[q][0], m[q][1]), 2 * mul(m[q][0], m[q][2]), 2 * mul(m[q][1], m[q][2]));
    const long long W0 = mul(m[0][0], m[1][0]), W1 = mul(m[0][1], m[1][1]), W2 = mul(m[0][2], m[1][2]);
    const long long S = W0 + W1 + W2;
    put(2, 0, 2 * W2 - S, 2 * W1 - S, 2 * W0 - S);
    // J = Im(w_2 conj(w_1)), w_k = U_mu,k U_ek: U_e1 U_e2 (im_2 re_1 - re_2 im_1)
    fxacc j;
    fx_mac(j, row[8], row[4]);
    fx_mac(j, fx_neg(row[5]), row[7]);
    v[12] = fx_split(4 * mul(fx_res(j), fx_split(mul(row[1], row[2]))));
}

// ---- bins whose layers are solved in place ------------------------------------------------
// (quadratic densities, where every segment has its own, and production-height averaging)

// What the bins of one energy share: the air layer and W's entries.
struct FxAir {
    fx U[3][3];     // eigenvectors of the air layer
    fx row[9];      // its flavour rows (fx_rows)
    fx coef[13];    // fx_coefficients
    double rate[2];
};
struct FxW {
    fx c, s, cr, ci, sr, si;  // cos, sin of theta23; the same times e^{i delta}
};
CP3_HD FxW fx_w(const double* w) {
    return FxW{fx_split(fx_from_double(w[0])),        fx_split(fx_from_double(w[1])),
               fx_split(fx_from_double(w[0] * w[2])), fx_split(fx_from_double(w[0] * w[3])),
               fx_split(fx_from_double(w[1] * w[2])), fx_split(fx_from_double(w[1] * w[3]))};
}

// a x + (b + i c) y: a row of W on entries x, y of a vector in the rotated basis
CP3_HD cfx fx_flavour(fx a, fx b, fx c, cfx x, cfx y) {
    fxacc2 r, m;
    fx_mac(r, a, x.re), fx_mac(r, b, y.re), fx_mac(r, fx_neg(c), y.im);
    fx_mac(m, a, x.im), fx_mac(m, b, y.im), fx_mac(m, c, y.re);
    return cfx{fx_res(r), fx_res(m)};
}

// U v and U^T v, U real
CP3_HD void fx_apply(const fx U[3][3], cfx v[3]) {
    const fx R[9] = {U[0][0], U[0][1], U[0][2], U[1][0], U[1][1], U[1][2], U[2][0], U[2][1], U[2][2]};
    fx_rotate(R, v);
}
CP3_HD void fx_apply_transposed(const fx U[3][3], cfx v[3]) {
    const fx R[9] = {U[0][0], U[1][0], U[2][0], U[0][1], U[1][1], U[2][1], U[0][2], U[1][2], U[2][2]};
    fx_rotate(R, v);
}

// The amplitude of the segments 1..M in the rotated basis, G = B^T S_M B with B = S_{M-1}..S_1
// (G = 1 for M = 0), ready to be applied to vectors: Y = U_M^T B, whose columns start from the
// rows of U_1.  solve(l, k) gives segment l's layer.
struct FxAmplitude {
    cfx y[3][3];
    cfx e[2];
    fx U1[3][3];
    int M;
    CP3_HD void apply(cfx k[3]) const {
        if (M == 0) return;
        if (M == 1) {
            fx_apply_transposed(U1, k);
            fx_phase(e, k);
            fx_apply(U1, k);
        } else {
            fx_palindrome(y, e, k);
        }
    }
};

template <class Solve>
CP3_HD void fx_chain(Solve solve, const double* len, int M, const longlong2* trig, unsigned int& bad, FxAmplitude& g) {
    g.M = M;
    FxDet det;
    fx U[3][3];
#pragma unroll 1
    for (int l = 1; l <= M; l++) {
        FxClass n;
        solve(l, n);
        if (l == 1) {
#pragma unroll
            for (int j = 0; j < 2; j++)
#pragma unroll
                for (int i = 0; i < 3; i++) g.y[j][i] = cfx{n.U[j][i], fx{0, 0}};
        } else {
            fx R[3][3];
            fx_rotation(n.U, U, R);
#pragma unroll
            for (int j = 0; j < 2; j++) {
                fx_phase(g.e, g.y[j]);
                fx_apply(R, g.y[j]);
            }
        }
        fx_layer(n.rate, len[l], trig, g.e, bad, l < M ? &det : nullptr);
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int k = 0; k < 3; k++) U[i][k] = n.U[i][k];
    }
    if (M == 1) {
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int k = 0; k < 3; k++) g.U1[i][k] = U[i][k];
    } else if (M > 1) {
        fx_third_column(det, trig, g.y);
    }
}

// One bin; false where it needs the FP64 path.  load() gives the air layer, which is not asked
// for before the chain of the others is done.
template <class Solve, class Load>
CP3_HD bool fx_bin_inline(Solve solve, Load load, const FxW& w, const double* len, int M,
                          const longlong2* trig, long long P[4]) {
    unsigned int bad = 0;
    FxAmplitude g;
    if (M > 0) fx_chain(solve, len, M, trig, bad, g);
    const FxAir air = load();
    cfx e0[2];
    fx_layer(air.rate, len[0], trig, e0, bad);
    if (M == 0) {
        fx_one_layer(air.coef, e0, P);
        return (bad >> 20) == 0;
    }
#pragma unroll 1
    for (int j = 0; j < 2; j++) {  // initial flavours e, mu: S_0 W^+ column j
        cfx k[3];
#pragma unroll
        for (int i = 0; i < 3; i++)
            k[i] = j == 0 ? cfx{air.row[i], fx{0, 0}} : cfx{air.row[3 + i], fx_neg(air.row[6 + i])};
        fx_phase(e0, k);
        fx_apply(air.U, k);
        g.apply(k);
        P[2 * j] = fx_norm(k[0]);
        P[2 * j + 1] = fx_norm(fx_flavour(w.c, w.sr, w.si, k[1], k[2]));
    }
    return (bad >> 20) == 0;
}

// ---- production-height averaging ----------------------------------------------------------
// physics.hpp:997-1130: with the amplitude split over the air layer's eigenstates,
// A = sum_k e_k a_k b_k^+ (a_k = W G u_k, b_k = W u_k), each cross term of a probability is
// weighted by t_kq = sum over height bins of prob sinc(d w / 2) e^{i d m}, d = -(omega_k -
// omega_q), m and w the mid shift and the width of the bin's path lengths:
//   P(j -> i) = sum_k |a_ki|^2 |b_kj|^2
//               + 2 sum_{q<k} Re[conj(a_qi) a_ki  e_k conj(e_q) b_qj conj(b_kj) t_kq,j].
// The a_k are orthonormal, so the sum over i is 1 whatever the weights, and the rows e and mu
// are enough.

// math::defined_sinc (math.hpp:49-55) as the reference evaluates it (its abs() is the int one:
// the series branch for every |x| < 1).
CP3_HD fx fx_sinc(double x) {
    if (!(fabs(x) < 1.0)) return fx_split(fx_from_double(sin(x) / x));
    const fx X = fx_split(fx_scaled(x, 1023));
    fxacc a;
    fx_mac(a, X, X);
    const fx x2 = fx_res(a);
    fxacc b, c;
    fx_mac(b, x2, fx_split(38430716820228232LL));  // 1 / 120
    fx_mac(c, x2, fx_split(768614336404564651LL - fx_sum(b)));  // 1 / 6 - x^2 / 120
    return fx_split((1LL << 62) - fx_sum(c));
}

// Weights that are no distribution: the smallest s >= 0 for which the weights times 2^-s are at
// most 1 and add up to less than 5/4 (total, largest: of the magnitudes; the margin covers the sum's
// rounding); kFxNoScale where there is none, and the bin takes the FP64 path.
constexpr int kFxNoScale = -1;
CP3_HD int fx_weight_scale(double total, double largest) {
    constexpr double most = 1.2499999;
    if (!(total <= 1e30)) return kFxNoScale;
    if (largest <= 1.0 && total <= most) return 0;
    int et, el;
    const double mt = frexp(total, &et), ml = frexp(largest, &el);  // m 2^e, 1/2 <= m < 1
    if (mt <= 0.5 * most) et--;
    if (ml <= 0.5) el--;
    const int s = et > el ? et : el;
    return s > 0 ? s : 0;
}

// The sums t over some of a bin's heights (b0, b0 + step, ...), and the sums of the weights'
// magnitudes (54 fraction bits).  The products' leading and cross terms accumulate over the
// heights as they are, with the low words cut to 27 bits (2^-57): the cross terms of 20 heights
// stay below 2^63 and no sum is formed per height.
struct FxShift {
    long long hh[3][3][2] = {}, x[3][3][2] = {};  // [pair][initial flavour][re, im]
    unsigned long long total[3] = {};
    CP3_HD long long value(int q, int f, int c) const { return hh[q][f][c] * 4 + (x[q][f][c] >> 25); }
};

// prob, mid, wid: the height bins' probabilities of the three initial flavours (b-th at
// prob[f * flavour + b * stride]), their mid shifts and widths in km.  kScaled: flavour f's are
// taken times 2^-scale[f].
template <bool kScaled = false>
CP3_HD void fx_shift_sums(const double rate[2], int b0, int step, int nb, const double* prob, size_t flavour,
                          size_t stride, const double* mid, const double* wid, const longlong2* trig,
                          unsigned int& bad, FxShift& o, const int* scale = nullptr) {
    const double pr[2] = {rate[0] * M_PI, rate[1] * M_PI};
#pragma unroll 1
    for (int b = b0; b < nb; b += step) {
        const double h = -mid[b], w = wid[b];
        double weight[3];  // asked for before the phases, which cover their way (49 us against 51)
#pragma unroll
        for (int f = 0; f < 3; f++) weight[f] = prob[f * flavour + b * stride];
        cfx z[3];
        double x[3];
#pragma unroll
        for (int q = 0; q < 2; q++) {
            fx_sincos(fx_angle(rate[q], h, bad), trig, z[q].re, z[q].im);
            x[q] = pr[q] * w;
        }
        x[2] = x[1] - x[0];
        z[2] = fx_cmul(cfx{z[0].re, fx_neg(z[0].im)}, z[1]);
#pragma unroll
        for (int q = 0; q < 3; q++) {
            const fx s = fx_sinc(x[q]);
            fxacc r, m;
            fx_mac(r, s, z[q].re);
            fx_mac(m, s, z[q].im);
            z[q] = cfx{fx_res(r), fx_res(m)};
            z[q].re.l >>= 5;
            z[q].im.l >>= 5;
        }
#pragma unroll
        for (int f = 0; f < 3; f++) {
            const double p = weight[f];
            const long long pb = fx_bits(p) & 0x7fffffffffffffffLL;
            const int one = kScaled ? 1023 + scale[f] : 1023;  // exponent of the largest
            const bool above = pb > (long long)one << 52;      // or not a number
            if (above) bad |= 1u << 20;
            const long long pv = above ? 0 : fx_scaled(p, one);
            o.total[f] += (unsigned long long)(pv < 0 ? -pv : pv) >> 8;
            fx pf = fx_split(pv);
            pf.l >>= 5;
#pragma unroll
            for (int q = 0; q < 3; q++)
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    const fx v = c == 0 ? z[q].re : z[q].im;
                    fx_mad(o.hh[q][f][c], pf.h, v.h);
                    fx_mad(o.x[q][f][c], pf.h, v.l);
                    fx_mad(o.x[q][f][c], pf.l, v.h);
                }
        }
    }
}

// The rows e, mu of a_k = W G u_k; load() as above.
template <class Solve, class Load>
CP3_HD void fx_air_rows(Solve solve, Load load, const FxW& w, const double* len, int M,
                        const longlong2* trig, unsigned int& bad, cfx a[2][3]) {
    FxAmplitude g;
    fx_chain(solve, len, M, trig, bad, g);
    const FxAir air = load();
#pragma unroll 1
    for (int k = 0; k < 3; k++) {
        cfx v[3];
#pragma unroll
        for (int i = 0; i < 3; i++) v[i] = cfx{air.U[i][k], fx{0, 0}};
        g.apply(v);
        a[0][k] = v[0];
        a[1][k] = fx_flavour(w.c, w.sr, w.si, v[1], v[2]);
    }
}

// The same from a table of the layers.
CP3_HD void fx_air_rows(const FxColumn& t, const double* len, int M, const longlong2* trig, unsigned int& bad,
                        cfx a[2][3]) {
    if (M == 0) {  // G = 1: the air layer's own flavour rows
#pragma unroll
        for (int k = 0; k < 3; k++) {
            a[0][k] = cfx{t.extra(kFxV0 + k), fx{0, 0}};
            a[1][k] = cfx{t.extra(kFxV0 + 3 + k), t.extra(kFxV0 + 6 + k)};
        }
        return;
    }
    auto layer = [&](int l, cfx* f, FxDet* det) {
        const double rate[2] = {t.rate(l, 0), t.rate(l, 1)};
        fx_layer(rate, len[l], trig, f, bad, det);
    };
    cfx y[3][3], e[2];
    if (M > 1) fx_columns(t, M, layer, trig, y);
    layer(M, e, nullptr);
#pragma unroll 1
    for (int k = 0; k < 3; k++) {
        cfx v[3];
#pragma unroll
        for (int i = 0; i < 3; i++) v[i] = cfx{t.rot(0, 3 * i + k), fx{0, 0}};  // U_1^T u_k
        if (M > 1)
            fx_palindrome(y, e, v);
        else
            fx_phase(e, v);
        fx_rows_of(t, v, a[0][k], a[1][k]);
    }
}

// Weights (as scaled) that add up to more than 5/4 leave the range of the factors t.
CP3_HD void fx_check_weights(const unsigned long long total[3], unsigned int& bad) {
#pragma unroll
    for (int f = 0; f < 3; f++)
        if (total[f] > (5ULL << 52)) bad |= 1u << 20;
}

// One averaged bin's probabilities of the initial flavour j, from these rows, the air layer's
// own (fx_rows) and its rates, and j's shift factors t: base[i] + 2 cross[i] is that of j -> i,
// i = e, mu, and cross is proportional to t.  The tau row's products follow from the others': the
// columns of W U_0 are orthonormal.
CP3_HD void fx_average(int j, const cfx a[2][3], const fx row[9], const double rate[2], double air_km,
                       const longlong2* trig, const cfx t[3], unsigned int& bad, long long base[2],
                       long long cross[2]) {
    cfx e[3];  // e_k conj(e_q) of the pairs (1,0), (2,0), (2,1)
    fx_layer(rate, air_km, trig, e, bad);
    e[2] = fx_cmul(cfx{e[0].re, fx_neg(e[0].im)}, e[1]);
    const int hi[3] = {1, 2, 2}, lo[3] = {0, 0, 1};
    fxacc2 s[2], x[2];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const int h = hi[k], l = lo[k];
        // |b_k|^2 and b_q conj(b_k)
        fxacc er, en;
        fx_mac(er, row[h], row[l]);
        fx_mac(en, row[k], row[k]);
        const cfx m = fx_cmul(cfx{row[3 + h], fx_neg(row[6 + h])}, cfx{row[3 + l], row[6 + l]});
        const long long mn = fx_norm(cfx{row[3 + k], row[6 + k]});
        const cfx c = j == 0   ? cfx{fx_res(er), fx{0, 0}}
                      : j == 1 ? m
                               : cfx{fx_split(-fx_sum(er) - fx_value(m.re)), fx_neg(m.im)};
        const fx norm = fx_split(j == 0 ? fx_sum(en) : j == 1 ? mn : (1LL << 62) - fx_sum(en) - mn);
        const cfx f = fx_cmul(t[k], fx_cmul(e[k], c));
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const cfx q = a[i][l];
            const cfx d = fx_cmul(cfx{q.re, fx_neg(q.im)}, a[i][h]);  // conj(a_qi) a_ki
            fx_mac(s[i], fx_split(fx_norm(a[i][k])), norm);
            fx_mac(x[i], d.re, f.re);
            fx_mac(x[i], fx_neg(d.im), f.im);
        }
    }
#pragma unroll
    for (int i = 0; i < 2; i++) {
        base[i] = fx_sum(s[i]);
        cross[i] = fx_sum(x[i]);
    }
}
CP3_HD void fx_average(int j, const cfx a[2][3], const fx row[9], const double rate[2], double air_km,
                       const longlong2* trig, const cfx t[3], unsigned int& bad, long long P[2]) {
    long long cross[2];
    fx_average(j, a, row, rate, air_km, trig, t, bad, P, cross);
#pragma unroll
    for (int i = 0; i < 2; i++) P[i] += 2 * cross[i];
}

}  // namespace cp3
