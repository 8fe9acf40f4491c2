// FFT mat-vec y = b - (1/M) F^-1[ G~ . F(pad(alpha x)) ]  on sm_100a.
//
// Replaces cdmlib/produitfftmatvectopt.f:3-121 (full box) and
// cdmlib/produitfftmatvect3.f:2-127 (Tabdip indirection), with the driver's
// `xi = polarisa . xr` step (cdmlib/inverserigopt.f:68-80) fused into the first
// pass.  The padded grid (X,Y,Z) = (2nx,2ny,2nz) is never materialised in full:
//
//   pass 1  fwd_x : read AoS x (3 per site) and alpha, FFT along x of the nx
//                   nonzeros padded to X              -> B1[r][c][k<nz][j<ny][X]
//   pass 2  fwd_y : FFT along y of the ny nonzeros     -> B2[r][c][k<nz][Y][X]
//   pass 3  zconv : FFT along z of the nz nonzeros, 3x3 symmetric multiply by
//                   the parity-compressed G~, inverse FFT along z, keep k<nz
//                                                     -> B2 (in place)
//   pass 4  inv_y : inverse FFT along y, keep j<ny     -> B1
//   pass 5  inv_x : inverse FFT along x, keep i<nx, y = b - v/M (AoS)
//
// Every pass loads its lines straight into the registers of the first FFT
// pass (the zero half of the padding is never read) and stores from the
// registers of the last one (the cropped half is never written); shared memory
// holds the tile between the inner FFT passes only.
//
// Order along X in B1 and B2: the frequencies qx = t and X - t lie side by
// side, at 2 t and 2 t + 1 (t = 0: qx = 0 and nx, which are their own
// mirrors).  Both see the same spectrum values up to the sign of xy and xz,
// which the x passes take out by storing component x of the mirrored one
// negated (S G S v with S = diag(-1, 1, 1)), so the y and z passes read one
// column of G~ for two columns of data.  In FP64 the two are neighbouring
// 16-byte elements; in FP32 they form one 16-byte element (cpair: both real
// parts, both imaginary parts), on which sums take one packed instruction
// for two values.  The x passes' butterflies j and X/R - j hold the
// frequencies t and X - t together, so a thread that does both writes or
// reads whole pairs.
//
// The compressed spectrum: G(r) on the circulant grid is even (xx,yy,zz) or odd
// (xy in x,y; xz in x,z; yz in y,z) under q -> (L - q) mod L along each axis
// (zero planes at nx,ny,nz, cdmlib/calculgreenfft.f:29-35), so its DFT has the
// same parity and only q in [0, L/2] per axis is stored, z fastest so that
// what a column of zconv needs is contiguous:
//   Gc[qy][qx][c6][qz], dims (ny+1, nx+1, 6, nz+1), c6 = xx,xy,xz,yy,yz,zz.
#pragma once
#include "fft_tile.cuh"
#include "reduce.cuh"

namespace ifdda {

struct MvGeom {
    int nx, ny, nz;     // lattice
    int X, Y, Z;        // padded FFT grid
    long N;             // nx*ny*nz
    long b1_rhs;        // elements of B1 per right-hand side: 3*nz*ny*X
    long b2_rhs;        // elements of B2 per right-hand side: 3*nz*Y*X
    long gc_comp;       // octant sites (nx+1)(ny+1)(nz+1): elements of one compressed G~ component
};

// polarisability modes
enum { ALPHA_NONE = 0, ALPHA_ISO = 1, ALPHA_FULL = 2 };

template <class T> struct MvArgs {
    using C = cplx<T>;
    MvGeom g;
    const C* x;          // input vectors, AoS, per rhs stride xstride
    const C* b;          // subtrahend vectors (may alias y)
    C* y;                // output vectors
    long xstride;        // complex elements between right-hand sides
    int amode;
    const C* alpha;      // ISO: alpha[d]; FULL: alpha[d + nmax*(a + 3*b)]
    long nmax;
    const int* tabdip;   // lattice -> 1-based dipole (null: identity)
    C* B1;
    C* B2;
    const C* Gc;         // compressed spectrum
    const C* twx;
    const C* twy;
    const C* twz;
    const int* status;   // per rhs: nonzero -> skip (solve finished)
    T inv_m;             // 1 / (X Y Z)
    int zvar, yvar;      // tile variants of zconv and of the y passes (MvTiles V)
    // Ragged batch (objects of different lattices, spacings and wavelengths
    // on one common box): per right-hand side, its object's spectrum and the
    // offsets of its polarisability (dipoles) and Tabdip (box sites) in the
    // concatenated alpha / tabdip arrays.  Null: one object for every rhs.
    const C* const* gc_r;
    const long* alpha_off;
    const long* tab_off;
    __device__ __forceinline__ const int* tab_of(int rhs) const { return tab_off ? tabdip + tab_off[rhs] : tabdip; }
    __device__ __forceinline__ const C* alpha_of(int rhs) const { return alpha_off ? alpha + alpha_off[rhs] : alpha; }
};

// Tile shapes: lines per block, threads per block and the register cap of
// each pass, with what they measured on B200.
//  * x passes: about 16 KB of shared memory (8 KB below length 64, where a
//    small lattice would otherwise leave SMs without a block).  FP32 keeps to 80
//    registers: at 96 the 1024 blocks of a 64^3 grid no longer fit the SMs at
//    once, and the solver's passes took 24.9 instead of 18.5 us;
//  * y passes: 16 columns of 16 bytes from length 64 on, 8 below and for V = 1
//    (FP64 there and back at 64^3 34.5 against 36.6 us; 8 leave a small
//    lattice more blocks).  Up to length 16 a column is one thread's: 16
//    columns (8 x 8 x 8, 8 right-hand sides: 8.6 us a product against 9.0 with
//    8 and 9.2 with 32), and 32 up to length 8 (64 x 2 x 64 in FP64 17.8 us
//    with 8, 14.6 with 16, 13.2 with 32);
//  * zconv: 8 columns of 16 bytes, rows of 128 bytes, from length 12 to 160.  4
//    columns (V = 1 from length 64 to 128) and 2 give more and smaller blocks,
//    but their narrower rows cost more than that: FP64 at 64^3 43.5, 47.5 and
//    65 us, FP32 27.9, 29.5 and 40.5 us.  Longer columns no longer fit 112 KB, so
//    that two blocks share an SM: V = 0 takes 4 at 192 and 256 (FP32 also at
//    320) and 2 beyond; V = 1, without the spectrum in shared memory, 8 up to 256,
//    4 at 320 and 384 (FP32 also at 512) and 2 beyond.
//    From 160 on two passes need 150 to 250 registers a thread, which leaves 6
//    to 12 warps per SM; there V = 1 takes three passes of small radices at 80
//    registers and reads the spectrum where it uses it (L2), so that 24 warps
//    fit: FP32 at 192^3 1.21 -> 0.89 ms.  Below, where two passes leave 12 warps
//    or more, three were slower (FP64 at 64^3 57.9 against 45.2 us: the extra
//    round trip through shared memory).
//    Up to length 8 a column is one thread's, with no shared memory in
//    between, and a block takes 32 columns (64 at length 2), at length 10 16:
//    with 8 columns and two passes most threads had no work.  Product of
//    256x256x1 in FP64 66.1 -> 33.7 us, 128x128x2 x4 70.4 -> 43.0, 128x128x4 x2
//    55.2 -> 43.8, 256x256x5 192.7 -> 130.9; in FP32 37.5 -> 25.0, 42.4 -> 30.0,
//    33.9 -> 30.9, 97.4 -> 67.0.
// Register caps of the y passes and of zconv's small middles (RK up to 5): 102
// (five warps per quarter SM; 84 for first radices up to 8 and at length 20)
// instead of 128: 12 right-hand sides of 48x40x32 in FP64 5.51 -> 5.24 ms a
// solve, 75x45x29 x2 86.7 -> 84.9 us a mat-vec; 128x128x16 x2 183.7 us a mat-vec
// in FP64 with 84, 187.4 with 102 and 193.5 with 128; 40x40x20 20.2 us with 84,
// 19.3 with 102, x8 76.7 and 77.6.  One pass takes what three times L points
// need (128x128x2 x4 in FP64 45.9 us with 84, which spills, 42.8 with 102 or 128).
// The variants are compiled for lengths of 64 and more; the tile chooser
// (tune_tiles) times both on the caller's grid and keeps one per grid.  The
// two agree to rounding.  Below length 160 V = 1 is for lattices whose wider
// tiles leave SMs without a block: products of 16x32x32 13.3 -> 12.3 us (FP32
// 11.5 -> 10.8), 32^3 in FP32 13.8 -> 12.6, 1x64x64 14.2 -> 11.8 (FP32 13.2 ->
// 12.2); from 40^3 or from several right-hand sides on V = 0 is as good or
// better (64^3 80.0 against 85.5 us, FP32 43.7 against 45.5).
//
// Tried without gain and left out: B2 stored in column tiles (z rows no longer
// a power of two apart), a persistent zconv that copies the next row's input
// under the current one (FP64 at 64^3 49 against 43.5 us), right-hand sides and
// column slabs run through the passes in groups that fit L2.
constexpr int tile_variants(int L) { return L >= 64 ? 2 : 1; }
template <class T, int L, int V = 0> struct MvTiles {
    using E = typename yz_elem<T>::type;
    static constexpr int S = (int)sizeof(cplx<T>);
    static constexpr int SE = (int)sizeof(E);
    static constexpr int SMEM_X = L >= 64 ? 16384 : 8192;
    static constexpr int TLX = clamp_pow2(SMEM_X / (3 * (L + 1) * S), 1, 16);
    static constexpr int TLY = L <= 8 ? 32 : L <= 16 || (V == 0 && L >= 64) ? 16 : 8;
    static constexpr int NBX = 3 * TLX, NBY = TLY;
    // x tile: points contiguous with one pad word every 16, line pitch = 8 (mod 16)
    static constexpr int lpitch() {
        int p = L + L / 16 + 1;
        while (p % 16 != 8) p++;
        return p;
    }
    static constexpr int LP = lpitch();
    static constexpr int round32(int t, int hi) {
        t = (t + 31) / 32 * 32;
        return t > hi ? hi : t;
    }
    // blocks per SM asked of the compiler so that it keeps to about cap
    // registers: a quarter of the SM holds 512 registers for each lane of its warps
    static constexpr int minblocks(int nt, int cap) {
        int m = 4 * (512 / cap) / (nt / 32);
        if (m * nt > 2048) m = 2048 / nt;
        return m < 1 ? 1 : (m > 32 ? 32 : m);
    }
    // x passes: radix of the last forward (first inverse) pass, its
    // butterflies per line and pairs of them (j, NJ - j)
    static constexpr int NPX = plan_len(L, PLAN_X);
    static constexpr int RX = plan_radix(L, NPX - 1, PLAN_X), NJX = L / RX, NJP = (NJX + 1) / 2;
    static constexpr int NTX = round32(NPX > 2 || NBX * NJP > NBX * (L / plan_radix(L, 0, PLAN_X))
                                           ? NBX * NJP : NBX * (L / plan_radix(L, 0, PLAN_X)), 512);
    // y passes: one butterfly of the first radix per thread
    static constexpr int RY = plan_radix(L, 0, PLAN_Y);
    static constexpr int NTY = round32(NBY * (L / RY), 512);
    // zconv: first radix, middle radix (the last of the plan), groups of the
    // middle per column
    // V = 1 from length 160 on: three small radices, and the spectrum read
    // from L2 where it is used instead of through shared memory
    static constexpr bool ZSMALL = V == 1 && L >= 160;
    static constexpr int PZ = ZSMALL ? PLAN_Z3 : PLAN_Z;
    static constexpr int NPZ = plan_len(L, PZ);
    static constexpr int RZ = plan_radix(L, 0, PZ), RK = plan_radix(L, NPZ - 1, PZ), NJZ = L / RK;
    // Tiles of 8 columns need no padding: 8 lanes of 16 bytes fill the banks.
    // With fewer, the butterflies j, j + 1 of the middle (RK a power of two)
    // must lie an odd number of points apart.
    static constexpr int log2i(int v) { return v <= 1 ? 0 : 1 + log2i(v / 2); }
    static constexpr bool RKP2 = RK == 2 || RK == 4 || RK == 8;
    static constexpr int zpadsh(int tl) { return tl >= 8 ? 0 : (RKP2 ? log2i(2 * RK) : RK == 12 ? 2 : 4); }
    static constexpr int zpadoff(int tl) { return tl >= 8 || !RKP2 ? 0 : RK; }
    static constexpr int zspan(int tl) { return zpadsh(tl) ? L + ((L + zpadoff(tl)) >> zpadsh(tl)) : L; }
    // G~ slice: columns of the tile (pairs share one) and one for qx = nx;
    // pitch of a column in W elements, a multiple of 16 bytes, chosen so that
    // neighbouring columns fall into different banks
    static constexpr int NQ = L / 2 + 1;
    static constexpr int gcols(int tl) { return S == 8 ? tl : tl / 2; }
    static constexpr int gpitch() {
        int g = 6 * NQ;
        if (S == 8) {
            while (g % 8 != 4) g++;
        } else {
            while (g % 8 != 2 && g % 8 != 6) g++;
        }
        return g;
    }
    static constexpr int GST = gpitch();
    static constexpr size_t zbytes(int tl) {
        return (size_t)L * S + (size_t)zspan(tl) * 3 * tl * SE + (ZSMALL ? 0 : (size_t)(gcols(tl) + 1) * GST * S);
    }
    static constexpr int ztile() {
        int tl = NPZ == 1 ? (L == 2 ? 64 : 32) : L == 10 ? 16 : V == 1 && !ZSMALL ? 4 : 8;
        while (tl > 2 && zbytes(tl) > 112 * 1024) tl /= 2;
        return tl;
    }
    static constexpr int TLZ = ztile(), NBZ = 3 * TLZ, TCZ = gcols(TLZ);
    static_assert(TLZ >= 2, "a zconv tile holds whole pairs");
    static constexpr int NTZ = ZSMALL || NPZ == 1 ? round32(TLZ * NJZ, 512) : round32(NBZ * (L / RZ) > TLZ * NJZ ? NBZ * (L / RZ) : TLZ * NJZ, 512);
    // L2 prefetch size of the column reads of zconv and the y passes (rows of
    // 32 to 256 bytes that neighbouring blocks read at the same time)
    static constexpr int ZPF = 256;
    using LayX = Layout<1, LP, false, 4>;
    using LayY = Layout<NBY, 1, true>;
    using LayZ = Layout<NBZ, 1, true, zpadsh(TLZ), zpadoff(TLZ)>;
    static constexpr int MINBX = minblocks(NTX, S == 8 ? 80 : (RX > 8 ? 128 : 102));
    static constexpr int MINBY = minblocks(NTY, RY == 32 ? 168 : 102);
    static constexpr int MINBZ = minblocks(NTZ, ZSMALL ? 84 : NPZ == 1 ? (L == 2 ? 84 : L == 4 ? 128 : L == 6 ? 168 : 248) : RK >= 10 ? 248 : (RZ == 32 || RK > 5 ? 168 : (RZ == 16 || L == 40 ? 102 : 84)));
    static constexpr size_t smem_x = (size_t)L * S + (size_t)NBX * LP * S;
    static constexpr size_t smem_y = (size_t)L * S + (size_t)L * NBY * SE;
    static constexpr size_t smem_z = zbytes(TLZ);
    static_assert(smem_z <= 227 * 1024 && smem_y <= 227 * 1024 && smem_x <= 227 * 1024, "tile above the SM's shared memory");
};

// asynchronous global -> shared copy of 16 bytes
__device__ __forceinline__ void cp_async16(void* dst_smem, const void* src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst_smem);
    asm volatile("cp.async.cg.shared.global.L2::256B [%0], [%1], 16;\n" ::"r"(d), "l"(src));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

template <class C> __device__ __forceinline__ C* smem_base() {
    extern __shared__ __align__(16) unsigned char ifdda_smem[];
    return reinterpret_cast<C*>(ifdda_smem);
}

// ---- pass 1 ---------------------------------------------------------------
// The mat-vec input: Pre::value(e) returns element e = 3 d + c of the vector
// to multiply.  PreNone reads it; a solver's Pre may instead form it from its
// own vectors (storing the result) and accumulate ND dot products, which the
// x pass leaves as per-block partial sums.  value() is called exactly once per
// element, except with a full polarisability tensor (three calls per
// element), which only PreNone supports.
template <class T> struct PreNone {
    static constexpr int ND = 0;
    const cplx<T>* x;
    double2 acc[1];
    __device__ __forceinline__ void bind(const MvArgs<T>& a, int rhs) { x = a.x + rhs * a.xstride; }
    template <class C> __device__ __forceinline__ C value(int e) { return __ldg(x + e); }
};

// Element offsets inside one right-hand side's vectors and scratch fit in 32
// bits for every compiled FFT length L (at most 3 (L/2)^3 dipole components
// and 3 (L/2) L^2 grid points, 3.9e8 at length 640; checked where the lengths
// are listed), and so do those of a full polarisability tensor of up to 2^31 / 9
// dipoles, so the pass functors index with int from per-block base pointers;
// the fields they need are copied by value.
template <class T, bool TAB, class Pre> struct FwdXLoad {
    static constexpr bool GLOBAL = true, HALF = true;  // points p >= nx are the padding
    const int* tab;
    const cplx<T>* alpha;
    int amode, nmax, nx;
    mutable Pre pre;
    int site0, nl, tl;
    template <class C> __device__ __forceinline__ C load(int b, int p) const {
        const int c = b / tl, jl = b - c * tl;
        if (jl >= nl) return czero<C>();
        const int site = site0 + jl * nx + p;
        int d = site;
        if (TAB) {
            const int t = __ldg(tab + site);
            if (t == 0) return czero<C>();
            d = t - 1;
        }
        if (amode == ALPHA_ISO) return cmul(__ldg(alpha + d), pre.template value<C>(3 * d + c));
        if (amode == ALPHA_FULL) {
            C acc = czero<C>();
#pragma unroll
            for (int q = 0; q < 3; q++)
                acc = cadd(acc, cmul(__ldg(alpha + d + nmax * (c + 3 * q)), pre.template value<C>(3 * d + q)));
            return acc;
        }
        return pre.template value<C>(3 * d + c);
    }
};

// Frequencies of a pair of butterflies (jA = jp, jB) of radix R on a line of
// length L = R NJ: butterfly j holds j + r NJ, r < R.  For jp > 0, jB = NJ - jp
// holds the mirrors: r of one is R - 1 - r of the other.  jp = 0 and (NJ even)
// jB = NJ / 2 hold their own: r and R - r (0 and R / 2 pair up as t = 0), and
// r and R - 1 - r.  NJ odd: jp = 0 has no jB.
template <int NJ> __device__ __forceinline__ int pair_jb(int jp) { return jp == 0 ? NJ / 2 : NJ - jp; }

// one element pair t of a B1 row: first = frequency t, second = X - t
__device__ __forceinline__ void pair_store(float2* row, int t, float2 f, float2 s) {
    reinterpret_cast<cpair*>(row)[t] = cpair{make_float2(f.x, s.x), make_float2(f.y, s.y)};
}
__device__ __forceinline__ void pair_store(double2* row, int t, double2 f, double2 s) {
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(row + 2 * t), "d"(f.x), "d"(f.y), "d"(s.x), "d"(s.y)
                 : "memory");
}
__device__ __forceinline__ void pair_load(const float2* row, int t, float2& f, float2& s) {
    const cpair v = reinterpret_cast<const cpair*>(row)[t];
    f = make_float2(v.re.x, v.im.x);
    s = make_float2(v.re.y, v.im.y);
}
__device__ __forceinline__ void pair_load(const double2* row, int t, double2& f, double2& s) {
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
                 : "=d"(f.x), "=d"(f.y), "=d"(s.x), "=d"(s.y)
                 : "l"(row + 2 * t)
                 : "memory");
}

// Last forward pass of an x tile: smem (or, for a one-pass plan, src) -> B1
// pairs.  base: row (c = 0, k, j0); nl valid rows; cstride: elements between
// components.
template <class C, int L, class TT, class Src>
__device__ __forceinline__ void x_store_pairs(const C* sm, const C* tw, const Src& src, C* base, int nl, int cstride) {
    constexpr int R = TT::RX, NJ = TT::NJX, NJP = TT::NJP, NT = TT::NTX, TL = TT::TLX;
    using Lay = typename TT::LayX;
    constexpr int ITEMS = TT::NBX * NJP, PER = (ITEMS + NT - 1) / NT;
#pragma unroll
    for (int q = 0; q < PER; q++) {
        const int u = threadIdx.x + q * NT;
        if (!(PER * NT == ITEMS || u < ITEMS)) continue;
        const int b = u / NJP, jp = u % NJP;
        const int c = b / TL, jl = b - c * TL;
        if (jl >= nl) continue;
        const int jb = pair_jb<NJ>(jp);
        const bool self = jp == 0;
        C A[R], B[R];
#pragma unroll
        for (int r = 0; r < R; r++) {
            if constexpr (TT::NPX == 1) {
                A[r] = 2 * r >= R ? czero<C>() : src.template load<C>(b, r);
                B[r] = czero<C>();
            } else {
                A[r] = sm[Lay::addr(jp + r * NJ, b)];
                B[r] = sm[Lay::addr(jb + r * NJ, b)];
                if (r > 0) {
                    A[r] = cmul(A[r], tw[jp * r]);
                    B[r] = cmul(B[r], tw[jb * r]);
                }
            }
        }
        Dft<R, +1, C>::run(A);
        Dft<R, +1, C>::run(B);
        C* row = base + c * cstride + jl * L;
        const typename elem_traits<C>::T sx = c == 0 ? -1 : 1;
#pragma unroll
        for (int r = 0; r < R / 2; r++) {
            const C own = r == 0 ? A[R / 2] : cscale(A[(R - r) % R], sx);  // t = 0 keeps its sign
            const C mir = cscale(B[R - 1 - r], sx);
            pair_store(row, jp + r * NJ, A[r], self ? own : mir);
        }
        if (NJ % 2 == 0 || !self) {
#pragma unroll
            for (int r = 0; r < R / 2; r++)
                pair_store(row, jb + r * NJ, B[r], cscale(self ? B[R - 1 - r] : A[R - 1 - r], sx));
        }
    }
}

// First inverse pass of an x tile: B1 pairs -> smem (or, for a one-pass plan, dst)
template <class C, int L, class TT, class Dst>
__device__ __forceinline__ void x_load_pairs(C* sm, const Dst& dst, const C* base, int nl, int cstride) {
    constexpr int R = TT::RX, NJ = TT::NJX, NJP = TT::NJP, NT = TT::NTX, TL = TT::TLX;
    using Lay = typename TT::LayX;
    constexpr int ITEMS = TT::NBX * NJP, PER = (ITEMS + NT - 1) / NT;
#pragma unroll
    for (int q = 0; q < PER; q++) {
        const int u = threadIdx.x + q * NT;
        if (!(PER * NT == ITEMS || u < ITEMS)) continue;
        const int b = u / NJP, jp = u % NJP;
        const int c = b / TL, jl = b - c * TL;
        const int jb = pair_jb<NJ>(jp);
        const bool self = jp == 0, has_b = NJ % 2 == 0 || !self;
        const typename elem_traits<C>::T sx = c == 0 ? -1 : 1;
        C A[R], B[R], sa[R / 2], sb[R / 2];
        const C* row = base + c * cstride + jl * L;
#pragma unroll
        for (int r = 0; r < R / 2; r++) {
            A[r] = B[r] = sa[r] = sb[r] = czero<C>();
            if (jl < nl) {
                pair_load(row, jp + r * NJ, A[r], sa[r]);
                if (has_b) pair_load(row, jb + r * NJ, B[r], sb[r]);
            }
        }
#pragma unroll
        for (int r = R / 2; r < R; r++) {
            const C own = r == R / 2 ? sa[0] : cscale(sa[R - r], sx);
            const C mir = cscale(sb[R - 1 - r], sx);
            A[r] = self ? own : mir;
            B[r] = cscale(self ? sb[R - 1 - r] : sa[R - 1 - r], sx);
        }
        Dft<R, -1, C>::run(A);
        Dft<R, -1, C>::run(B);
#pragma unroll
        for (int r = 0; r < R; r++) {
            if constexpr (TT::NPX == 1) {
                if (2 * r < R) dst.template store<C>(b, r, A[r]);
            } else {
                sm[Lay::addr(jp * R + r, b)] = A[r];
                if (has_b) sm[Lay::addr(jb * R + r, b)] = B[r];
            }
        }
    }
    if constexpr (TT::NPX > 1) __syncthreads();
}

template <class T, int L, bool TAB, class TT = MvTiles<T, L>, class Pre = PreNone<T>>
__global__ void __launch_bounds__(TT::NTX, TT::MINBX) k_fwd_x(const MvArgs<T> a, const Pre pre, const MvRed red) {
    using C = cplx<T>;
    constexpr int TL = TT::TLX, NB = TT::NBX, NT = TT::NTX, NP = TT::NPX;
    const int rhs = blockIdx.z;
    C* tw = smem_base<C>();
    C* sm = tw + L;
    const int nx = a.g.nx, ny = a.g.ny, nz = a.g.nz;
    const int j0 = blockIdx.x * TL, k = blockIdx.y;
    const int nl = min(TL, ny - j0);
    load_twiddles<C, L, NT>(tw, a.twx);
    pdl_wait();
    pdl_trigger();
    if (a.status && a.status[rhs]) return;
    using Src = FwdXLoad<T, TAB, Pre>;
    Src src{a.tab_of(rhs), a.alpha_of(rhs), a.amode, (int)a.nmax, nx, pre, k * nx * ny + j0 * nx, nl, TL};
    src.pre.bind(a, rhs);
    C* base = a.B1 + rhs * a.g.b1_rhs + ((long)k * ny + j0) * L;
    if constexpr (NP > 1)
        stockham_range<C, L, NB, NT, +1, typename TT::LayX, false, NP - 1, 0, 1, Src, SmemIO, PLAN_X>(sm, tw, src,
                                                                                                       SmemIO{});
    x_store_pairs<C, L, TT>(sm, tw, src, base, nl, nz * ny * L);
    if constexpr (Pre::ND > 0)
        block_partial<NT, Pre::ND>(src.pre.acc,
                                   red.ppart + (((long)rhs * gridDim.y + k) * red.gxs + blockIdx.x) * Pre::ND);
}

// ---- pass 2 and 4 ---------------------------------------------------------
// DIR=+1: B1 (ny rows) -> B2 (Y rows);  DIR=-1: B2 (Y rows) -> B1 (ny rows)
template <class E, int DIR, int PF = 0> struct YLoad {
    static constexpr bool GLOBAL = true, HALF = DIR > 0;  // forward: rows >= ny are padding
    const E* src;   // first column of the tile
    int pitch, nv;  // elements between rows, valid columns
    template <class C> __device__ __forceinline__ C load(int b, int p) const {
        return b < nv ? ld_l2pf<PF>(src + p * pitch + b) : czero<C>();
    }
};
template <class E, int DIR> struct YStore {
    static constexpr bool GLOBAL = true, HALF = DIR < 0;  // inverse: keep rows < ny
    E* dst;
    int pitch, nv;
    template <class C> __device__ __forceinline__ void store(int b, int p, C v) const {
        if (b < nv) dst[p * pitch + b] = v;
    }
};

template <class T, int L, int DIR, class TT = MvTiles<T, L>>
__global__ void __launch_bounds__(TT::NTY, TT::MINBY) k_pass_y(const MvArgs<T> a) {
    using E = typename TT::E;
    using W = cplx<T>;
    constexpr int TL = TT::TLY, NT = TT::NTY, V = TT::SE / TT::S;  // complex values per element
    const int rhs = blockIdx.z / 3, c = blockIdx.z - 3 * rhs;
    W* tw = smem_base<W>();
    E* sm = reinterpret_cast<E*>(tw + L);
    const int XE = a.g.X / V, ny = a.g.ny, nz = a.g.nz;
    const int i0 = blockIdx.x * TL, k = blockIdx.y;
    load_twiddles<W, L, NT>(tw, a.twy);
    pdl_wait();
    pdl_trigger();
    if (a.status && a.status[rhs]) return;
    const int nv = min(TL, XE - i0);
    E* b1 = reinterpret_cast<E*>(a.B1 + rhs * a.g.b1_rhs) + ((long)c * nz + k) * ny * XE + i0;
    E* b2 = reinterpret_cast<E*>(a.B2 + rhs * a.g.b2_rhs) + ((long)c * nz + k) * L * XE + i0;
    YLoad<E, DIR, TT::ZPF> src{DIR > 0 ? b1 : b2, XE, nv};
    YStore<E, DIR> dst{DIR > 0 ? b2 : b1, XE, nv};
    fft_tile<E, L, TL, NT, DIR, typename TT::LayY, YLoad<E, DIR, TT::ZPF>, YStore<E, DIR>, PLAN_Y>(sm, tw, src, dst);
}

// ---- pass 3 -----------------------------------------------------------------
// lines b = c * TL + il: component c of column il
template <class E, int TL, int PF = 0> struct ZLoad {
    static constexpr bool GLOBAL = true, HALF = true;  // rows >= nz are padding
    const E* base;  // first column of the tile
    int rs, comp;   // elements between z rows and between components
    int nv;         // valid columns
    template <class C> __device__ __forceinline__ C load(int b, int p) const {
        const int c = b / TL, il = b - c * TL;
        return ld_l2pf<PF>(base + c * comp + p * rs + min(il, nv - 1));  // columns beyond the last are not stored
    }
};
template <class E, int TL> struct ZStore {
    static constexpr bool GLOBAL = true, HALF = true;  // keep z rows < nz
    E* base;
    int rs, comp, nv;
    template <class C> __device__ __forceinline__ void store(int b, int p, C v) const {
        const int c = b / TL, il = b - c * TL;
        if (il < nv) base[c * comp + p * rs + il] = v;
    }
};

// acc + g v with g = s (g.x + i g.y), s = +-1 folded into the products' signs
__device__ __forceinline__ double2 gfma(double2 acc, double2 g, double s, double2 v) {
    const double gx = s * g.x, gy = s * g.y;
    return make_double2(fma(gx, v.x, fma(-gy, v.y, acc.x)), fma(gx, v.y, fma(gy, v.x, acc.y)));
}
__device__ __forceinline__ cpair gfma(cpair acc, float2 g, float s, cpair v) {
    const float gx = s * g.x, gy = s * g.y;
    const float2 gx2 = make_float2(gx, gx), gy2 = make_float2(gy, gy), ng2 = make_float2(-gy, -gy);
    return cpair{fma2(gx2, v.re, fma2(ng2, v.im, acc.re)), fma2(gx2, v.im, fma2(gy2, v.re, acc.im))};
}
__device__ __forceinline__ double2 gmul(double2 g, double2 v) {
    return make_double2(fma(g.x, v.x, -g.y * v.y), fma(g.x, v.y, g.y * v.x));
}
__device__ __forceinline__ cpair gmul(float2 g, cpair v) {
    const float2 gx2 = make_float2(g.x, g.x), gy2 = make_float2(g.y, g.y), ng2 = make_float2(-g.y, -g.y);
    return cpair{fma2(gx2, v.re, mul2(ng2, v.im)), fma2(gx2, v.im, mul2(gy2, v.re))};
}
// acc + s g v with one g per value of the pair (the column t = 0: qx = 0, nx)
__device__ __forceinline__ cpair gfma2(cpair acc, float2 g0, float2 g1, float s, cpair v) {
    const float2 gx = make_float2(s * g0.x, s * g1.x), gy = make_float2(s * g0.y, s * g1.y);
    return cpair{fma2(gx, v.re, fma2(make_float2(-gy.x, -gy.y), v.im, acc.re)),
                 fma2(gx, v.im, fma2(gy, v.re, acc.im))};
}

// v with its sign bits flipped where f is the sign bit (0: v)
__device__ __forceinline__ float2 flip(float2 v, unsigned f) {
    return make_float2(__uint_as_float(__float_as_uint(v.x) ^ f), __uint_as_float(__float_as_uint(v.y) ^ f));
}

// v <- G v for the RK points j + r NJ of one column; g: its slice [c6][qz].
// Spectral mirrors: z beyond nz flips xz and yz, the row Y - qy xy and yz
// (component x of a mirrored column is stored negated, so xy and xz need no
// flip for X - qx).  MY: the row is a mirrored one (1), is not (0), or is where
// my is the sign bit (-1).
template <class E, int L, int RK, int MY, class W>
__device__ __forceinline__ void zmultiply(E (&v)[3][RK], const W* g, unsigned my, int j) {
    using T = typename elem_traits<E>::T;
    constexpr int NJ = L / RK, NQ = L / 2 + 1;
    const T sy = MY == 1 ? T(-1) : T(1);
#pragma unroll
    for (int r = 0; r < RK; r++) {
        const int p = j + r * NJ;
        // at 2 p = L the odd components vanish, either sign will do
        const bool mir = RK % 2 == 0 ? 2 * r >= RK : 2 * p > L;
        const W* gq = g + (mir ? L - p : p);
        const T sz = mir ? T(-1) : T(1);
        const E x = v[0][r], y = v[1][r], z = v[2][r];
        W gxy = gq[NQ], gxz = gq[2 * NQ], gyz = gq[4 * NQ];
        if constexpr (MY < 0) {
            gxy = flip(gxy, my);
            gyz = flip(gyz, my);
        }
        v[0][r] = gfma(gfma(gmul(gq[0], x), gxy, sy, y), gxz, sz, z);
        v[1][r] = gfma(gfma(gmul(gq[3 * NQ], y), gxy, sy, x), gyz, sy * sz, z);
        v[2][r] = gfma(gfma(gmul(gq[5 * NQ], z), gxz, sz, x), gyz, sy * sz, y);
    }
}
// the same for an FP32 pair whose two values have columns of their own (t = 0)
template <int L, int RK>
__device__ __forceinline__ void zmultiply_ends(cpair (&v)[3][RK], const float2* g0, const float2* g1, unsigned my,
                                               int j) {
    constexpr int NJ = L / RK, NQ = L / 2 + 1;
#pragma unroll
    for (int r = 0; r < RK; r++) {
        const int p = j + r * NJ;
        const bool mir = 2 * p > L;
        const int q = mir ? L - p : p;
        const float sz = mir ? -1.f : 1.f;
        const cpair x = v[0][r], y = v[1][r], z = v[2][r];
        const cpair o = czero<cpair>();
        const float2 xy0 = flip(g0[q + NQ], my), xy1 = flip(g1[q + NQ], my);
        const float2 yz0 = flip(g0[q + 4 * NQ], my), yz1 = flip(g1[q + 4 * NQ], my);
        v[0][r] = gfma2(gfma2(gfma2(o, g0[q], g1[q], 1.f, x), xy0, xy1, 1.f, y), g0[q + 2 * NQ], g1[q + 2 * NQ], sz, z);
        v[1][r] = gfma2(gfma2(gfma2(o, g0[q + 3 * NQ], g1[q + 3 * NQ], 1.f, y), xy0, xy1, 1.f, x), yz0, yz1, sz, z);
        v[2][r] = gfma2(gfma2(gfma2(o, g0[q + 5 * NQ], g1[q + 5 * NQ], 1.f, z), g0[q + 2 * NQ], g1[q + 2 * NQ], sz, x),
                        yz0, yz1, sz, y);
    }
}

// Forward z transform (passes 0 .. n-2 of the plan), then in registers: the
// last forward pass, the 3x3 multiply and the first pass of the inverse
// transform run on the reversed plan, so the inverse starts from the values
// the forward one ended with (its pass 0 reads exactly the points
// j + r L/R the forward last pass produced), then inverse passes 1 .. n-1.
//
// Bound by latency at 12 warps per SM: at 64^3 the FP64 pipe, shared memory and
// instruction issue are each 35-40% busy.  Against one complex value per
// thread and element, a slice of the spectrum per column and 2.06e7 warp
// instructions: FP64 58.1 -> 42.9 us (1.54e7), FP32 35.2 -> 26.9 us (1.95e7 ->
// 0.98e7: packed sums, one spectrum value for two columns, no work on the
// padding's zeros).
// Grid (2 right-hand side + mirror row, column tile, qy): the blocks that read
// one slice of the spectrum run together, so a batch takes that slice from
// HBM once (L2 serves the rest).
template <class T, int L, class TT = MvTiles<T, L>>
__global__ void __launch_bounds__(TT::NTZ, TT::MINBZ) k_zconv(const MvArgs<T> a) {
    using E = typename TT::E;
    using W = cplx<T>;
    using LZ = typename TT::LayZ;
    constexpr int TL = TT::TLZ, NB = TT::NBZ, NT = TT::NTZ, TC = TT::TCZ, GST = TT::GST;
    constexpr int NP = TT::NPZ;
    constexpr int RK = TT::RK;                 // last forward radix = first inverse radix
    constexpr int NJ = TT::NJZ;                // butterflies per line in that pass
    constexpr int NG = TL * NJ;                // (column, butterfly) groups
    constexpr int PERM = (NG + NT - 1) / NT;
    constexpr int V = TT::SE / TT::S;          // complex values per element
    // hm = 1 takes row Y - qy (which exists for 0 < qy < ny only)
    const int rhs = (int)blockIdx.x >> 1, hm = (int)blockIdx.x & 1;
    W* tw = smem_base<W>();
    E* sm = reinterpret_cast<E*>(tw + L);
    W* gs = reinterpret_cast<W*>(sm + LZ::span(L) * NB);
    const int nx = a.g.nx, ny = a.g.ny, nz = a.g.nz, Y = a.g.Y, XE = a.g.X / V;
    const int i0 = blockIdx.y * TL;
    const int qy = blockIdx.z;                    // 0 .. ny
    if (hm && !(qy > 0 && qy < ny)) {
        pdl_wait();
        return;
    }
    const int t0 = i0 * V / 2;           // first pair of the tile
    load_twiddles<W, L, NT>(tw, a.twz);
    // the tile's columns of the compressed spectrum (contiguous each) are
    // copied into shared memory while the forward transform runs; the last
    // one is qx = nx, the partner of t = 0
    const W* gbase = (a.gc_r ? a.gc_r[rhs] : a.Gc) + (long)qy * (nx + 1) * (6 * TT::NQ);
    if constexpr (!TT::ZSMALL) {
        constexpr int CH = 6 * TT::NQ * (int)sizeof(W) / 16;
        static_assert(6 * TT::NQ * sizeof(W) % 16 == 0 && GST * sizeof(W) % 16 == 0, "16-byte copies");
        const char* src = reinterpret_cast<const char*>(gbase + (long)t0 * (6 * TT::NQ));
        char* dst = reinterpret_cast<char*>(gs);
        if constexpr (2 * CH <= NT) {  // several columns at a time
            for (int e = threadIdx.x; e < min(TC, nx - t0) * CH; e += NT)
                cp_async16(dst + e / CH * (GST * (int)sizeof(W)) + e % CH * 16, src + 16 * e);
            if (t0 == 0 && (int)threadIdx.x < CH)
                cp_async16(dst + TC * (GST * (int)sizeof(W)) + 16 * threadIdx.x,
                           src + (long)nx * (CH * 16) + 16 * threadIdx.x);
        } else {
#pragma unroll
            for (int col = 0; col <= TC; col++) {
                const int qx = col < TC ? t0 + col : nx;
                if (!(col < TC ? qx < nx : t0 == 0)) continue;
                const char* cs = src + (long)(qx - t0) * (CH * 16) + 16 * threadIdx.x;
                char* cd = dst + col * (GST * (int)sizeof(W)) + 16 * threadIdx.x;
#pragma unroll
                for (int ch = 0; ch < CH; ch += NT)
                    if (ch + NT <= CH || ch + (int)threadIdx.x < CH) cp_async16(cd + 16 * ch, cs + 16 * ch);
            }
        }
        cp_async_commit();
    }
    // the spectrum and the twiddles are constant: only B2 waits for the y pass
    pdl_wait();
    pdl_trigger();
    if (a.status && a.status[rhs]) {
        if constexpr (!TT::ZSMALL) cp_async_wait_all();
        return;
    }
    const int rs = Y * XE, comp = nz * rs, nv = min(TL, XE - i0);
    E* B2 = reinterpret_cast<E*>(a.B2 + rhs * a.g.b2_rhs) + (long)(hm ? Y - qy : qy) * XE + i0;
    const ZLoad<E, TL, TT::ZPF> zload{B2, rs, comp, nv};
    const ZStore<E, TL> zstore{B2, rs, comp, nv};
    if constexpr (NP > 1) {
        stockham_pass<E, L, TT::RZ, 1, NB, NT, +1, LZ, ZLoad<E, TL, TT::ZPF>, SmemIO, false>(sm, tw, zload, SmemIO{});
        if constexpr (!TT::ZSMALL && NP == 2) cp_async_wait_all();
        __syncthreads();
        stockham_range<E, L, NB, NT, +1, LZ, false, NP - 1, 1, TT::RZ, SmemIO, SmemIO, TT::PZ>(sm, tw, SmemIO{},
                                                                                              SmemIO{});
    }
    if constexpr (!TT::ZSMALL && NP != 2) {
        cp_async_wait_all();
        __syncthreads();
    }
    const unsigned my = hm ? 0x80000000u : 0u;
    // ---- fused middle: read, transform, multiply, transform (registers) ----
    E v[PERM][3][RK];
#pragma unroll
    for (int q = 0; q < PERM; q++) {
        const int g = threadIdx.x + q * NT;
        if (!(PERM * NT == NG || g < NG)) continue;
        const int il = g % TL, j = g / TL;
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const int b = c * TL + il;
#pragma unroll
            for (int r = 0; r < RK; r++) {
                const int p = j + r * NJ;
                if constexpr (NP == 1) {
                    // (no load for a column beyond the last: the one before is being written)
                    v[q][c][r] = 2 * p >= L || il >= nv ? czero<E>() : zload.template load<E>(b, p);
                } else if constexpr (read_split<LZ>(NJ, RK)) {
                    v[q][c][r] = sm[LZ::addr(j, b) + LZ::pidx(r * NJ) * LZ::PS];
                } else {
                    v[q][c][r] = sm[LZ::addr(p, b)];
                }
            }
            if constexpr (NJ > 1) {
                // forward last pass: Ns = NJ, k = j, twiddle w^(j r)
#pragma unroll
                for (int r = 1; r < RK; r++) v[q][c][r] = cmul(v[q][c][r], tw[j * r]);
            }
            Dft<RK, +1, E>::run(v[q][c]);
        }
        if (il < nv) {
            const int t = V == 2 ? il : il >> 1;  // column of the slice
            const bool ends = V == 2 ? t0 + t == 0 : (t0 == 0 && il == 1);
            if constexpr (V == 2) {
                const W* g0 = TT::ZSMALL ? gbase + (long)(t0 + t) * (6 * TT::NQ) : gs + t * GST;
                // The whole tile of t = 0 takes the form with two columns, and the row's sign is a
                // value: no warp runs two forms, and the code, which a small grid's few waves
                // fetch about as often as they run it, is shorter (zconv of 16^3 x8 4.28 -> 3.74 us,
                // 64^3 20.9 -> 19.9).  FP64, whose columns are one each, keeps a form per row sign
                // (35.2 against 35.7 us at 64^3).
                if (t0 == 0)
                    zmultiply_ends<L, RK>(v[q], g0,
                                          !ends ? g0 : TT::ZSMALL ? gbase + (long)nx * (6 * TT::NQ) : gs + TC * GST, my,
                                          j);
                else zmultiply<E, L, RK, -1>(v[q], g0, my, j);
            } else {
                const W* gcol = TT::ZSMALL ? gbase + (long)(ends ? nx : t0 + t) * (6 * TT::NQ) : gs + (ends ? TC : t) * GST;
                if (hm) zmultiply<E, L, RK, 1>(v[q], gcol, my, j);
                else zmultiply<E, L, RK, 0>(v[q], gcol, my, j);
            }
        }
        // inverse pass 0 of the reversed plan: Ns = 1, inputs j + r NJ, no twiddles
#pragma unroll
        for (int c = 0; c < 3; c++) Dft<RK, -1, E>::run(v[q][c]);
    }
    if constexpr (NP > 1) __syncthreads();  // every read of the tile is done
#pragma unroll
    for (int q = 0; q < PERM; q++) {
        const int g = threadIdx.x + q * NT;
        if (!(PERM * NT == NG || g < NG)) continue;
        const int il = g % TL, j = g / TL;
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const int b = c * TL + il;
#pragma unroll
            for (int r = 0; r < RK; r++) {
                const int o = j * RK + r;
                if constexpr (NP == 1) {
                    if (2 * o < L) zstore.template store<E>(b, o, v[q][c][r]);
                } else if constexpr (write_split<LZ>(NJ, 1, RK)) {
                    sm[LZ::addr(j * RK, b) + LZ::pidx(r) * LZ::PS] = v[q][c][r];
                } else {
                    sm[LZ::addr(o, b)] = v[q][c][r];
                }
            }
        }
    }
    if constexpr (NP > 1) {
        __syncthreads();
        stockham_range<E, L, NB, NT, -1, LZ, true, NP, 1, RK, SmemIO, ZStore<E, TL>, TT::PZ>(sm, tw, SmemIO{},
                                                                                            zstore);
    }
}

// ---- pass 5 -----------------------------------------------------------------
// The mat-vec output: Epi::elem(e, y) sees every stored element y of the
// result (e = 3 d + c) and may accumulate ND dot products; the last block of
// the grid then holds them, with the NDP partials of the first x pass, and
// calls Epi::finish.
//
// The vectors that a tile's last pass reads are known from the start: b and the
// Epi's own (Epi::ahead) are asked into L2 before the transform, which then
// runs while they come from DRAM (FP64 solves: 64^3 4.92 -> 4.80 ms, 12
// right-hand sides of an ellipsoid on 48x40x32 5.35 -> 5.28 ms).  ahead() is
// called for the first element of a dipole; the three components of one lie
// within 48 bytes.
template <class C> __device__ __forceinline__ void prefetch_l2(const C* p) {
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}
struct EpiNone {
    static constexpr int ND = 0, NDP = 0;
    double2 acc[1];
    template <class T> __device__ __forceinline__ void bind(const MvArgs<T>&, int) {}
    __device__ __forceinline__ void ahead(int) const {}
    template <class C> __device__ __forceinline__ void elem(int, C) {}
    __device__ __forceinline__ void finish(int, const double2*) {}
};

template <class T, bool TAB, class Epi> struct InvXStore {
    static constexpr bool GLOBAL = true, HALF = true;  // keep points < nx
    const int* tab;
    const cplx<T>* bv;
    cplx<T>* yv;
    T inv_m;
    int nx, site0, nl, tl;
    mutable Epi epi;
    template <class C> __device__ __forceinline__ void store(int b, int p, C v) const {
        const int c = b / tl, jl = b - c * tl;
        if (jl >= nl) return;
        const int site = site0 + jl * nx + p;
        int d = site;
        if (TAB) {
            const int t = __ldg(tab + site);
            if (t == 0) return;
            d = t - 1;
        }
        // b is read at an element before this thread writes y there (b may be y)
        const C y = csub(__ldg(bv + 3 * d + c), cscale(v, inv_m));
        yv[3 * d + c] = y;
        epi.elem(3 * d + c, y);
    }
};

template <class T, int L, bool TAB, class Epi, class TT = MvTiles<T, L>>
__global__ void __launch_bounds__(TT::NTX, TT::MINBX) k_inv_x(const MvArgs<T> a, const Epi epi, const MvRed red) {
    using C = cplx<T>;
    constexpr int TL = TT::TLX, NB = TT::NBX, NT = TT::NTX;
    const int rhs = blockIdx.z;
    C* tw = smem_base<C>();
    C* sm = tw + L;
    const int nx = a.g.nx, ny = a.g.ny, nz = a.g.nz;
    const int j0 = blockIdx.x * TL, k = blockIdx.y;
    const int nl = min(TL, ny - j0);
    load_twiddles<C, L, NT>(tw, a.twx);
    pdl_wait();
    if (a.status && a.status[rhs]) return;
    const C* base = a.B1 + rhs * a.g.b1_rhs + ((long)k * ny + j0) * L;
    InvXStore<T, TAB, Epi> dst{a.tab_of(rhs), a.b + rhs * a.xstride, a.y + rhs * a.xstride, a.inv_m, nx,
                               k * nx * ny + j0 * nx, nl, TL, epi};
    dst.epi.bind(a, rhs);
    // one prefetch per dipole with a Tabdip, per 128 bytes without
    constexpr int STEP = TAB ? 1 : 128 / (3 * (int)sizeof(C));
    for (int i = threadIdx.x * STEP; i < nl * nx; i += NT * STEP) {
        const int d = TAB ? __ldg(dst.tab + dst.site0 + i) - 1 : dst.site0 + i;
        if (d < 0) continue;
        prefetch_l2(dst.bv + 3 * d);
        dst.epi.ahead(3 * d);
    }
    x_load_pairs<C, L, TT>(sm, dst, base, nl, nz * ny * L);
    if constexpr (TT::NPX > 1)
        stockham_range<C, L, NB, NT, -1, typename TT::LayX, true, TT::NPX, 1, TT::RX, SmemIO, InvXStore<T, TAB, Epi>,
                       PLAN_X>(sm, tw, SmemIO{}, dst);
    __syncthreads();  // the block's part of y is written: the next kernel may read it through ldg
    pdl_trigger();
    if constexpr (Epi::ND > 0) {
        double2 tot[Epi::ND + Epi::NDP];
        if (reduce_rows<NT, Epi::ND, Epi::NDP>(dst.epi.acc, tot, rhs, blockIdx.x, k, gridDim.x, gridDim.y, red) &&
            threadIdx.x == 0)
            dst.epi.finish(rhs, tot);
    }
}

}  // namespace ifdda
