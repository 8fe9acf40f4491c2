// Shared-memory Stockham FFT on a tile of NB independent lines of length L.
//
// Each pass of radix R combines R sub-transforms of length Ns into one of
// length Ns * R (autosort Stockham, natural-order output):
//     v[r] = x[j + r L/R] * w^(DIR * (j mod Ns) * r * L / (Ns R)),  r < R
//     v    = DFT_R(v, DIR)
//     x[(j / Ns) Ns R + (j mod Ns) + r Ns] = v[r]
// An inner pass keeps its butterflies in registers across a barrier, so the
// transform runs in place; a pass that reads from global memory or writes to
// it has no such hazard and no barrier of its own (after a transform that ends
// in global memory, a caller that reuses the tile synchronises first).  DIR = +1 is exp(+i 2 pi jk / L) (the reference's
// "forward" convention for G and x, cdmlib/calculgreenfft.f:16,76-99), DIR = -1
// the inverse; both unnormalised.  L may be any product of 2, 3 and 5.
//
// The first pass may read its inputs straight from global memory (Src::GLOBAL)
// and the last pass may write straight to global memory (Dst::GLOBAL), so a
// transform costs one shared-memory round trip less at each end.  With
// Src::HALF the upper half of the input is known to be zero (the padding of
// the circulant embedding) and is neither loaded nor stored; with Dst::HALF
// only the first half of the output is written (the crop).
//
// Shared-memory layout: point p of line b at sm[p * PS + b * BS].  With
// BFAST the butterflies of consecutive threads belong to consecutive lines
// (use with BS = 1: lines contiguous in global memory, e.g. the y and z axes);
// otherwise consecutive threads take consecutive points of one line (PS = 1,
// e.g. the x axis).
#pragma once
#include "cplx.cuh"

namespace ifdda {

// radices 8, 4, 2, 3, 5 in that order of preference
__host__ __device__ constexpr int pick_radix_basic(int rem) {
    return rem % 8 == 0 ? 8 : rem % 4 == 0 ? 4 : rem % 2 == 0 ? 2 : rem % 3 == 0 ? 3 : rem % 5 == 0 ? 5 : 0;
}
__host__ __device__ constexpr int passes_basic(int rem) {
    int n = 0;
    while (rem > 1) {
        const int r = pick_radix_basic(rem);
        if (r == 0) return 1000;
        rem /= r;
        n++;
    }
    return n;
}
// radix of the pass that has `rem` = L / Ns points left to combine: the
// first pass takes 16 where that saves a whole pass (one shared-memory round
// trip less; the first pass needs no table twiddles), otherwise 8, 4, 2, 3, 5
__host__ __device__ constexpr int pick_radix(int rem, bool first = false) {
    return (first && rem % 16 == 0 && 1 + passes_basic(rem / 16) < passes_basic(rem)) ? 16 : pick_radix_basic(rem);
}
__host__ __device__ constexpr bool smooth235(int L) {
    if (L < 1) return false;
    while (L % 2 == 0) L /= 2;
    while (L % 3 == 0) L /= 3;
    while (L % 5 == 0) L /= 5;
    return L == 1;
}
__host__ __device__ constexpr int clamp_pow2(int v, int lo, int hi) {
    int p = 1;
    while (p * 2 <= v && p * 2 <= hi) p *= 2;
    return p < lo ? lo : p;
}
// Radices with a register butterfly (Dft<R> below).
__host__ __device__ constexpr bool has_dft(int r) {
    return r == 2 || r == 3 || r == 4 || r == 5 || r == 6 || r == 8 || r == 10 || r == 12 || r == 16 || r == 32;
}
// Plans of the mat-vec passes (policy 0 is the general rule above):
//  PLAN_Z: one pass up to 8, two up to 384, the second (whose butterflies hold
//      all three components of a column in registers) of at most 8 points up
//      to 256 and 12 above: 16-byte elements at three times 8 points take 96
//      registers.  Factors 5 go into the first pass: with a five-point middle
//      zconv of 256x256x5 took 103 us in FP64 instead of 40 (46.5, 22.4 in
//      FP32), of 128x128x20 43.3 instead of 37.7 (22.3, 19.9);
//  PLAN_Z3: three passes with small radices: one shared-memory round trip more
//      per direction, for half the registers and twice the warps;
//  PLAN_Y: two passes up to 512;
//  PLAN_X: the last radix is even and at most 12, since a thread of the last
//      forward (first inverse) pass holds two butterflies at once.
enum { PLAN_ANY = 0, PLAN_Z = 1, PLAN_Y = 2, PLAN_X = 3, PLAN_Z3 = 4 };
struct RadixPlan {
    int r[3];
};
__host__ __device__ constexpr RadixPlan plan_table(int L, int policy) {
    switch (policy) {
    case PLAN_Z:
        switch (L) {
        case 4: return {{4}};
        case 6: return {{6}};
        case 8: return {{8}};
        case 10: return {{5, 2}};
        case 12: return {{4, 3}};
        case 16: return {{4, 4}};
        case 20: return {{10, 2}};
        case 24: return {{8, 3}};
        case 32: return {{8, 4}};
        case 40: return {{10, 4}};
        case 48: return {{16, 3}};
        case 64: return {{16, 4}};
        case 80: return {{16, 5}};
        case 96: return {{16, 6}};
        case 128: return {{16, 8}};
        case 160: return {{32, 5}};
        case 192: return {{32, 6}};
        case 256: return {{32, 8}};
        case 320: return {{32, 10}};
        case 384: return {{32, 12}};
        case 512: return {{16, 8, 4}};
        case 640: return {{16, 8, 5}};
        }
        break;
    case PLAN_Z3:
        switch (L) {
        case 160: return {{8, 5, 4}};
        case 192: return {{8, 6, 4}};
        case 256: return {{8, 8, 4}};
        case 320: return {{8, 10, 4}};
        case 384: return {{8, 12, 4}};
        case 512: return {{8, 16, 4}};
        case 640: return {{16, 10, 4}};
        }
        break;
    case PLAN_Y:
        switch (L) {
        case 6: return {{6}};
        case 10: return {{10}};
        case 12: return {{12}};
        case 16: return {{16}};
        case 20: return {{4, 5}};
        case 24: return {{8, 3}};
        case 32: return {{8, 4}};
        case 40: return {{8, 5}};
        case 48: return {{8, 6}};
        case 64: return {{8, 8}};
        case 80: return {{8, 10}};
        case 96: return {{16, 6}};
        case 128: return {{16, 8}};
        case 160: return {{16, 10}};
        case 192: return {{16, 12}};
        case 256: return {{16, 16}};
        case 320: return {{32, 10}};
        case 384: return {{32, 12}};
        case 512: return {{32, 16}};
        case 640: return {{16, 8, 5}};
        }
        break;
    case PLAN_X:
        switch (L) {
        case 4: return {{2, 2}};
        case 6: return {{3, 2}};
        case 8: return {{2, 4}};
        case 10: return {{5, 2}};
        case 12: return {{3, 4}};
        case 16: return {{4, 4}};
        case 20: return {{5, 4}};
        case 24: return {{3, 8}};
        case 32: return {{4, 8}};
        case 40: return {{5, 8}};
        case 48: return {{6, 8}};
        case 64: return {{8, 8}};
        case 80: return {{10, 8}};
        case 96: return {{16, 6}};
        case 128: return {{16, 8}};
        case 160: return {{16, 10}};
        case 192: return {{16, 12}};
        case 256: return {{4, 8, 8}};
        case 320: return {{5, 8, 8}};
        case 384: return {{16, 3, 8}};
        case 512: return {{8, 8, 8}};
        case 640: return {{10, 8, 8}};
        }
        break;
    }
    return {{0}};
}
__host__ __device__ constexpr int pick_radix_p(int L, int rem, bool first, int policy) {
    if (policy) {
        const RadixPlan t = plan_table(L, policy);
        int left = L;
        for (int q = 0; q < 3 && t.r[q] > 0; q++) {
            if (left == rem) return t.r[q];
            left /= t.r[q];
        }
    }
    return pick_radix(rem, first);
}
// The plan of L: radix of pass q (0-based) and number of passes.  A plan
// runs forward (q = 0 .. n-1) or reversed; any order of the radices is a
// valid Stockham transform, and the reversed plan lets an inverse transform
// start from the registers the forward transform ended with.
__host__ __device__ constexpr int plan_len(int L, int policy = 0) {
    int n = 0;
    bool first = true;
    for (int rem = L; rem > 1;) {
        const int r = pick_radix_p(L, rem, first, policy);
        if (r == 0) return -1;
        rem /= r;
        first = false;
        n++;
    }
    return n;
}
__host__ __device__ constexpr int plan_radix(int L, int q, int policy = 0) {
    int rem = L;
    bool first = true;
    for (int i = 0; i < q; i++) {
        rem /= pick_radix_p(L, rem, first, policy);
        first = false;
    }
    return pick_radix_p(L, rem, first, policy);
}
__host__ __device__ constexpr int plan_radix_dir(int L, int q, bool rev, int policy = 0) {
    return rev ? plan_radix(L, plan_len(L, policy) - 1 - q, policy) : plan_radix(L, q, policy);
}

// Exact mathematical constants used by the radix-3/5/8 butterflies.
#define IFDDA_SQRT3_2 0.86602540378443864676372317075294
#define IFDDA_SQRT1_2 0.70710678118654752440084436210485
#define IFDDA_C1_5 0.30901699437494742410229341718282   // cos(2 pi / 5)
#define IFDDA_C2_5 -0.80901699437494742410229341718282  // cos(4 pi / 5)
#define IFDDA_S1_5 0.95105651629515357211643933337938   // sin(2 pi / 5)
#define IFDDA_S2_5 0.58778525229247312916870595463907   // sin(4 pi / 5)

// Butterflies, in place on registers.  C is an FFT element (float2, double2
// or cpair); run_half assumes v[r] = 0 for r >= R / 2 (the padding), whose
// sums it leaves out.  Composite radices with coprime factors (6, 10, 12) use
// the prime-factor index maps, which need no inner twiddles.
template <int R, int DIR, class C> struct Dft;

template <int DIR, class C> struct Dft<2, DIR, C> {
    __device__ __forceinline__ static void run(C* v) {
        C a = v[0], b = v[1];
        v[0] = cadd(a, b);
        v[1] = csub(a, b);
    }
    __device__ __forceinline__ static void run_half(C* v) { v[1] = v[0]; }
};

template <int DIR, class C> struct Dft<3, DIR, C> {
    __device__ __forceinline__ static void run(C* v) {
        using T = typename elem_traits<C>::T;
        C t1 = cadd(v[1], v[2]);
        C t2 = cfma_s(v[0], t1, (T)-0.5);
        C t3 = csub(v[1], v[2]);
        const T s = DIR > 0 ? (T)IFDDA_SQRT3_2 : (T)-IFDDA_SQRT3_2;
        v[0] = cadd(v[0], t1);
        v[1] = cfma_i(t2, t3, s);
        v[2] = cfma_i(t2, t3, -s);
    }
};

template <int DIR, class C> struct Dft<4, DIR, C> {
    __device__ __forceinline__ static void run(C* v) {
        C s02 = cadd(v[0], v[2]), d02 = csub(v[0], v[2]);
        C s13 = cadd(v[1], v[3]), d13 = csub(v[1], v[3]);
        v[0] = cadd(s02, s13);
        v[2] = csub(s02, s13);
        v[1] = cadd_i<DIR>(d02, d13);
        v[3] = cadd_i<-DIR>(d02, d13);
    }
    __device__ __forceinline__ static void run_half(C* v) {
        C a = v[0], b = v[1];
        v[0] = cadd(a, b);
        v[2] = csub(a, b);
        v[1] = cadd_i<DIR>(a, b);
        v[3] = cadd_i<-DIR>(a, b);
    }
};

template <int DIR, class C> struct Dft<5, DIR, C> {
    __device__ __forceinline__ static void run(C* v) {
        using T = typename elem_traits<C>::T;
        const T c1 = (T)IFDDA_C1_5, c2 = (T)IFDDA_C2_5, s1 = (T)IFDDA_S1_5, s2 = (T)IFDDA_S2_5;
        C t1 = cadd(v[1], v[4]), t2 = cadd(v[2], v[3]);
        C t3 = csub(v[1], v[4]), t4 = csub(v[2], v[3]);
        C a1 = cfma_s(cfma_s(v[0], t1, c1), t2, c2);
        C a2 = cfma_s(cfma_s(v[0], t1, c2), t2, c1);
        C b1 = cfma_s(cscale(t3, s1), t4, s2);
        C b2 = cfma_s(cscale(t3, s2), t4, -s1);
        v[0] = cadd(v[0], cadd(t1, t2));
        v[1] = cadd_i<DIR>(a1, b1);
        v[4] = cadd_i<-DIR>(a1, b1);
        v[2] = cadd_i<DIR>(a2, b2);
        v[3] = cadd_i<-DIR>(a2, b2);
    }
};

// A x B points, A and B coprime: X[(n1 ka + n2 kb) mod R] from DFT_A over
// DFT_B of x[(B n1 + A n2) mod R]; ka = 1 mod A and 0 mod B, kb the other way
template <int A, int B, int DIR, class C> struct DftPfa {
    static constexpr int R = A * B;
    static constexpr int unit(int m, int n) {  // the multiple of n that is 1 mod m
        int q = n;
        while (q % m != 1) q += n;
        return q;
    }
    __device__ __forceinline__ static void run(C* v) {
        constexpr int ka = unit(A, B), kb = unit(B, A);
        C a[A][B];
#pragma unroll
        for (int n1 = 0; n1 < A; n1++) {
            C t[B];
#pragma unroll
            for (int n2 = 0; n2 < B; n2++) t[n2] = v[(B * n1 + A * n2) % R];
            Dft<B, DIR, C>::run(t);
#pragma unroll
            for (int n2 = 0; n2 < B; n2++) a[n1][n2] = t[n2];
        }
#pragma unroll
        for (int k2 = 0; k2 < B; k2++) {
            C t[A];
#pragma unroll
            for (int n1 = 0; n1 < A; n1++) t[n1] = a[n1][k2];
            Dft<A, DIR, C>::run(t);
#pragma unroll
            for (int k1 = 0; k1 < A; k1++) v[(k1 * ka + k2 * kb) % R] = t[k1];
        }
    }
    __device__ __forceinline__ static void run_half(C* v) {
#pragma unroll
        for (int r = R / 2; r < R; r++) v[r] = czero<C>();
        run(v);
    }
};
template <int DIR, class C> struct Dft<6, DIR, C> : DftPfa<2, 3, DIR, C> {};
template <int DIR, class C> struct Dft<10, DIR, C> : DftPfa<2, 5, DIR, C> {};
template <int DIR, class C> struct Dft<12, DIR, C> : DftPfa<4, 3, DIR, C> {};

template <int DIR, class C> struct Dft<8, DIR, C> {
    template <bool HALF> __device__ __forceinline__ static void go(C* v) {
        using T = typename elem_traits<C>::T;
        C e[4] = {v[0], v[2], v[4], v[6]};
        C o[4] = {v[1], v[3], v[5], v[7]};
        if constexpr (HALF) {
            Dft<4, DIR, C>::run_half(e);
            Dft<4, DIR, C>::run_half(o);
        } else {
            Dft<4, DIR, C>::run(e);
            Dft<4, DIR, C>::run(o);
        }
        const T h = (T)IFDDA_SQRT1_2;
        // w^1 = (1 + DIR i)/sqrt2, w^2 = DIR i, w^3 = (-1 + DIR i)/sqrt2
        const C o1 = cadd_i<DIR>(o[1], o[1]), o3 = cadd_i<-DIR>(o[3], o[3]);
        v[0] = cadd(e[0], o[0]);
        v[4] = csub(e[0], o[0]);
        v[1] = cfma_s(e[1], o1, h);
        v[5] = cfma_s(e[1], o1, -h);
        v[2] = cadd_i<DIR>(e[2], o[2]);
        v[6] = cadd_i<-DIR>(e[2], o[2]);
        v[3] = cfma_s(e[3], o3, -h);
        v[7] = cfma_s(e[3], o3, h);
    }
    __device__ __forceinline__ static void run(C* v) { go<false>(v); }
    __device__ __forceinline__ static void run_half(C* v) { go<true>(v); }
};

// 16 points as 4 x 4: DFT4 over the stride-4 subsequences, the inner twiddles
// w16^(n2 k1), then DFT4 across them; X[k1 + 4 k2]
#define IFDDA_COS_PI8 0.92387953251128675612818318939679  // cos(pi / 8)
#define IFDDA_SIN_PI8 0.38268343236508977172845998403040  // sin(pi / 8)
template <int DIR, class C> struct Dft<16, DIR, C> {
    template <bool HALF> __device__ __forceinline__ static void go(C* v) {
        using T = typename elem_traits<C>::T;
        C a[4][4];
#pragma unroll
        for (int n2 = 0; n2 < 4; n2++) {
            C t[4] = {v[n2], v[4 + n2], v[8 + n2], v[12 + n2]};
            if constexpr (HALF) Dft<4, DIR, C>::run_half(t);
            else Dft<4, DIR, C>::run(t);
#pragma unroll
            for (int k1 = 0; k1 < 4; k1++) a[n2][k1] = t[k1];
        }
        const T c = (T)IFDDA_COS_PI8, s = (T)IFDDA_SIN_PI8, h = (T)IFDDA_SQRT1_2;
        const T ds = DIR > 0 ? s : -s, dc = DIR > 0 ? c : -c, dh = DIR > 0 ? h : -h;
        // w^1 = c + i DIR s, w^2 = (1 + i DIR)/sqrt2, w^3 = s + i DIR c,
        // w^4 = i DIR, w^6 = (-1 + i DIR)/sqrt2, w^9 = -w^1
        a[1][1] = cmulk(a[1][1], c, ds);
        a[1][2] = cmulk(a[1][2], h, dh);
        a[1][3] = cmulk(a[1][3], s, dc);
        a[2][1] = cmulk(a[2][1], h, dh);
        a[2][3] = cmulk(a[2][3], -h, dh);
        a[3][1] = cmulk(a[3][1], s, dc);
        a[3][2] = cmulk(a[3][2], -h, dh);
        a[3][3] = cmulk(a[3][3], -c, -ds);
#pragma unroll
        for (int k1 = 0; k1 < 4; k1++) {
            // the factor w^4 = i DIR of a[2][2] goes into its two sums
            const C s02 = k1 == 2 ? cadd_i<DIR>(a[0][k1], a[2][k1]) : cadd(a[0][k1], a[2][k1]);
            const C d02 = k1 == 2 ? cadd_i<-DIR>(a[0][k1], a[2][k1]) : csub(a[0][k1], a[2][k1]);
            const C s13 = cadd(a[1][k1], a[3][k1]), d13 = csub(a[1][k1], a[3][k1]);
            v[k1] = cadd(s02, s13);
            v[k1 + 8] = csub(s02, s13);
            v[k1 + 4] = cadd_i<DIR>(d02, d13);
            v[k1 + 12] = cadd_i<-DIR>(d02, d13);
        }
    }
    __device__ __forceinline__ static void run(C* v) { go<false>(v); }
    __device__ __forceinline__ static void run_half(C* v) { go<true>(v); }
};

// 32 points as 2 x 16: DFT16 over the even and the odd points, the twiddles
// w32^k on the odd half, then DFT2 across; X[k] and X[k + 16]
#define IFDDA_COS_PI16 0.98078528040323044912618223613424   // cos(pi / 16)
#define IFDDA_SIN_PI16 0.19509032201612826784828486847702   // sin(pi / 16)
#define IFDDA_COS_3PI16 0.83146961230254523707878837761791  // cos(3 pi / 16)
#define IFDDA_SIN_3PI16 0.55557023301960222474283081394853  // sin(3 pi / 16)
template <int DIR, class C> struct Dft<32, DIR, C> {
    template <bool HALF> __device__ __forceinline__ static void go(C* v) {
        using T = typename elem_traits<C>::T;
        C e[16], o[16];
#pragma unroll
        for (int n = 0; n < 16; n++) {
            e[n] = v[2 * n];
            o[n] = v[2 * n + 1];
        }
        if constexpr (HALF) {
            Dft<16, DIR, C>::run_half(e);
            Dft<16, DIR, C>::run_half(o);
        } else {
            Dft<16, DIR, C>::run(e);
            Dft<16, DIR, C>::run(o);
        }
        // cos and sin of k pi / 16, k = 0..8 (k pi / 16 for k > 8 by symmetry)
        const T cs[9] = {(T)1, (T)IFDDA_COS_PI16, (T)IFDDA_COS_PI8, (T)IFDDA_COS_3PI16, (T)IFDDA_SQRT1_2,
                         (T)IFDDA_SIN_3PI16, (T)IFDDA_SIN_PI8, (T)IFDDA_SIN_PI16, (T)0};
#pragma unroll
        for (int k = 0; k < 16; k++) {
            // w32^k = cos(k pi/16) + i DIR sin(k pi/16)
            if (k == 8) {
                v[k] = cadd_i<DIR>(e[k], o[k]);
                v[k + 16] = cadd_i<-DIR>(e[k], o[k]);
                continue;
            }
            const T c = k <= 8 ? cs[k] : -cs[16 - k];
            const T sn = k <= 8 ? cs[8 - k] : cs[k - 8];
            const C t = k == 0 ? o[0] : cmulk(o[k], c, DIR > 0 ? sn : -sn);
            v[k] = cadd(e[k], t);
            v[k + 16] = csub(e[k], t);
        }
    }
    __device__ __forceinline__ static void run(C* v) { go<false>(v); }
    __device__ __forceinline__ static void run_half(C* v) { go<true>(v); }
};

// Source / destination that is the shared-memory tile itself.
struct SmemIO {
    static constexpr bool GLOBAL = false;
    static constexpr bool HALF = false;
    template <class C> __device__ C load(int, int) const { return C(); }
    template <class C> __device__ void store(int, int, C) const {}
};

// PADSH > 0 inserts one padding word every 2^PADSH points, so the strided
// writes of a radix-R pass (points j*R + r of consecutive j) spread over the
// shared-memory banks.
// PADOFF shifts where the padding words fall.
template <int PS_, int BS_, bool BFAST_, int PADSH_ = 0, int PADOFF_ = 0> struct Layout {
    static constexpr int PS = PS_, BS = BS_, PADSH = PADSH_, PADOFF = PADOFF_;
    static constexpr bool BFAST = BFAST_;
    // padded position of point p
    __host__ __device__ static constexpr int pidx(int p) { return PADSH ? p + ((p + PADOFF) >> PADSH) : p; }
    __device__ __forceinline__ static int addr(int p, int b) { return pidx(p) * PS + b * BS; }
    // points spanned by a line of length L (padding included)
    static constexpr int span(int L) { return PADSH ? L + ((L + PADOFF) >> PADSH) : L; }
};

// True when the padded positions of a butterfly's points j + r NJ (j < NJ,
// r < R) are pidx(j) + pidx(r NJ): the shared-memory address of every point
// is then the thread's base address plus a compile-time offset.
template <class Lay> constexpr bool read_split(int NJ, int R) {
    for (int j = 0; j < NJ; j++)
        for (int r = 0; r < R; r++)
            if (Lay::pidx(j + r * NJ) - Lay::pidx(j) != Lay::pidx(r * NJ)) return false;
    return true;
}
// The same for the outputs d + r Ns, d = (j / Ns) Ns R + j mod Ns, of a pass.
template <class Lay> constexpr bool write_split(int NJ, int Ns, int R) {
    for (int j = 0; j < NJ; j++) {
        const int d = (j / Ns) * Ns * R + j % Ns;
        for (int r = 0; r < R; r++)
            if (Lay::pidx(d + r * Ns) - Lay::pidx(d) != Lay::pidx(r * Ns)) return false;
    }
    return true;
}

// One Stockham pass.  tw[j] = exp(+2 pi i j / L) in shared memory.  SYNC: a pass
// that writes the tile ends in a barrier (otherwise the caller's next one does).
template <class C, int L, int R, int Ns, int NB, int NT, int DIR, class Lay, class Src, class Dst, bool SYNC = true>
__device__ __forceinline__ void stockham_pass(C* sm, const typename elem_traits<C>::W* tw, const Src& src,
                                              const Dst& dst) {
    using W = typename elem_traits<C>::W;
    const int tid = threadIdx.x;
    constexpr int NJ = L / R;
    constexpr int NBF = NB * NJ;
    constexpr int PER = (NBF + NT - 1) / NT;
    constexpr int TSTEP = L / (Ns * R);
    constexpr bool FIRST = Ns == 1, LAST = Ns * R == L;
    constexpr bool GIN = FIRST && Src::GLOBAL, GOUT = LAST && Dst::GLOBAL;
    constexpr bool RSPLIT = read_split<Lay>(NJ, R), WSPLIT = write_split<Lay>(NJ, Ns, R);
    // one butterfly: inputs, twiddles, transform
    const auto read = [&](C(&v)[R], int u) {
        const int b = Lay::BFAST ? u % NB : u / NJ;
        const int j = Lay::BFAST ? u / NB : u % NJ;
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int p = j + r * NJ;
            if (GIN) {
                // zero upper half: for an even radix p >= L/2 exactly when r >= R/2
                const bool zero = Src::HALF && (R % 2 == 0 ? 2 * r >= R : 2 * p >= L);
                v[r] = zero ? czero<C>() : src.template load<C>(b, p);
            } else if constexpr (RSPLIT) {
                v[r] = sm[Lay::addr(j, b) + Lay::pidx(r * NJ) * Lay::PS];
            } else {
                v[r] = sm[Lay::addr(p, b)];
            }
        }
        if (Ns > 1) {
            const int k = j % Ns;
#pragma unroll
            for (int r = 1; r < R; r++) {
                W w = tw[k * r * TSTEP];
                if (DIR < 0) w = cconj(w);
                v[r] = cmul(v[r], w);
            }
        }
        if constexpr (GIN && Src::HALF && R % 2 == 0) Dft<R, DIR, C>::run_half(v);
        else Dft<R, DIR, C>::run(v);
    };
    const auto write = [&](const C(&v)[R], int u) {
        const int b = Lay::BFAST ? u % NB : u / NJ;
        const int j = Lay::BFAST ? u / NB : u % NJ;
        const int k = j % Ns;
        const int d = (j / Ns) * Ns * R + k;
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int o = d + r * Ns;
            if (GOUT) {
                // last pass: o = j + r L/R; for an even radix o < L/2 exactly when r < R/2
                const bool keep = !Dst::HALF || (R % 2 == 0 ? 2 * r < R : 2 * o < L);
                if (keep) dst.template store<C>(b, o, v[r]);
            } else if constexpr (WSPLIT) {
                sm[Lay::addr(d, b) + Lay::pidx(r * Ns) * Lay::PS] = v[r];
            } else {
                sm[Lay::addr(o, b)] = v[r];
            }
        }
    };
    if constexpr (GIN || GOUT) {
        // the tile is only written or only read: one butterfly after the other, no barrier between
#pragma unroll
        for (int q = 0; q < PER; q++) {
            const int u = tid + q * NT;
            if (PER * NT == NBF || u < NBF) {
                C v[R];
                read(v, u);
                write(v, u);
            }
        }
    } else {
        C v[PER][R];
#pragma unroll
        for (int q = 0; q < PER; q++)
            if (PER * NT == NBF || tid + q * NT < NBF) read(v[q], tid + q * NT);
        __syncthreads();
#pragma unroll
        for (int q = 0; q < PER; q++)
            if (PER * NT == NBF || tid + q * NT < NBF) write(v[q], tid + q * NT);
    }
    if (!GOUT && SYNC) __syncthreads();
}

// Passes q in [q, Q1) of the plan (reversed when REV); Ns is the product of
// the radices of the passes before q.
template <class C, int L, int NB, int NT, int DIR, class Lay, bool REV, int Q1, int q, int Ns, class Src, class Dst,
          int PLAN = 0>
__device__ __forceinline__ void stockham_range(C* sm, const typename elem_traits<C>::W* tw, const Src& src,
                                               const Dst& dst) {
    if constexpr (q < Q1) {
        constexpr int R = plan_radix_dir(L, q, REV, PLAN);
        stockham_pass<C, L, R, Ns, NB, NT, DIR, Lay, Src, Dst>(sm, tw, src, dst);
        stockham_range<C, L, NB, NT, DIR, Lay, REV, Q1, q + 1, Ns * R, Src, Dst, PLAN>(sm, tw, src, dst);
    }
}

// Transform NB lines.  When the source is shared memory the caller must have
// synchronised after filling it; when the destination is shared memory the
// result may be read right after the call (the last pass ends in a barrier).
// The twiddle table must be resident before the second pass (the first pass
// uses none), so a caller may start filling it together with the first pass.
template <class C, int L, int NB, int NT, int DIR, class Lay, class Src = SmemIO, class Dst = SmemIO, int PLAN = 0>
__device__ __forceinline__ void fft_tile(C* sm, const typename elem_traits<C>::W* tw, const Src& src = Src(),
                                         const Dst& dst = Dst()) {
    static_assert(smooth235(L), "FFT length must be a product of 2, 3 and 5");
    stockham_range<C, L, NB, NT, DIR, Lay, false, plan_len(L, PLAN), 0, 1, Src, Dst, PLAN>(sm, tw, src, dst);
}

// shared-memory to shared-memory transform with lines fastest (LS >= NB)
template <class C, int L, int NB, int LS, int NT, int DIR>
__device__ __forceinline__ void tile_fft(C* sm, const C* tw) {
    fft_tile<C, L, NB, NT, DIR, Layout<LS, 1, true>>(sm, tw);
}

// copy the twiddle table for length L into shared memory
template <class C, int L, int NT>
__device__ __forceinline__ void load_twiddles(C* tws, const C* __restrict__ twg) {
    for (int j = threadIdx.x; j < L; j += NT) tws[j] = twg[j];
}

}  // namespace ifdda
