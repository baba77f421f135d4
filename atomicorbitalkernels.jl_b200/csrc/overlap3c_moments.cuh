// overlap3c_moments.cuh -- batched 3-center overlap of bases with f shells, templated on
// the element type (instantiated in overlap3c_moments_f32.cu / overlap3c_moments_f64.cu).
//
// Replaces batch_V_kernel! (src/integrals/kernels_3c.jl:12-162):
//   V_{mu nu lambda}(b) = int phi_mu(r - A_b) phi_nu(r - B_b) phi_lambda(r - C_b) dr.
// Per primitive triple the three Gaussians combine at Q = (aA + bB + cC)/q
// with prefactor c_a c_b c_c (pi/q)^{3/2} exp(-(ab|AB|^2 + ac|AC|^2 + bc|BC|^2)/q)
// (the reference's mu|AB|^2 + nu|PC|^2).  The sum over primitive triples is taken
// first, into moments, and the angular recursion runs once per block
// (moment3c.cuh).  The reference's aliased layout
// lin = c1 + (2la+1) c2 + (2la+1)(2lb+1) c3 (kernels_3c.jl:146-160) is applied when
// the blocks are written out.
//
// Two kernels per call, lane = batch element of a tile of 32 of one species triple:
//   k_moments3    units (segment of blocks, tile): the primitive triples of a block summed
//                 into its moments, written as one row of 32 lanes per moment.  A heavy
//                 block's triples are shared out over a CTA's warps.
//   k_transform3  units (panel, tile), a panel being a run of A shells with one B and one C
//                 shell: the CTA's warps run the recursions of its blocks, tasks (block,
//                 part of its components), into a shared-memory slab (one row per
//                 element), and stream the slab out; for every (j, k) the panel's whole run
//                 of i is contiguous in the output.
// Batches whose moments exceed kMoments3 go through in rounds.
//
// Bases with few primitives keep explicit E tables (pick3 in overlap3c_moments.cu).
//
// What bounds it (777 elements of a 32-function basis of two elements, s to f, up to 8
// primitives per shell; FP64, counters): k_moments3, 203 us, issues in 48 % of the cycles,
// held up by the exponentials' arithmetic and by the barriers of shared blocks.
// k_transform3, 262 us, issues in 13 % with 12 warps per SM: they wait at the barriers around
// a panel's tasks, for moments and for values spilled to local memory (f-f-f parts spill 3
// to 10 KB a thread, f-f-d up to 3, f-d-d up to 2.7, d-d-d 1), and for instructions, the
// recursions being straight-line code run once per (block, tile).  Whole call, against the
// routine with explicit E tables per triple and run-time loops: 3,815 -> 472 us in FP64,
// 3,120 -> 428 in FP32; 60 elements 2,280 -> 244 and 1,880 -> 216.  The output alone is 31
// and 16 us.
// Tried: the recursions run by one warp per panel without barriers (2,600 us: one f block is
// a long serial chain that holds up its whole panel); the moments summed in the same CTA as
// a phase of their own (805 us).  Why the slab: stores straight from the lanes (each to its own
// element) reach 0.18 T outputs/s whatever computes them: 230 us for 768 blocks of 32^3 in
// FP64, 67 us in rows of 96 bytes or more.
#pragma once

#include <algorithm>
#include <cstring>

#include "aok_internal.h"
#include "moment3c.cuh"

namespace aok {
namespace m3 {

constexpr int kThreads3 = 128;       // k_moments3
constexpr int kWarps3 = kThreads3 / 32;
constexpr int kMomCtas3 = 4;         // k_moments3: <= 128 registers
constexpr int64_t kMoments3 = 256 << 20;
constexpr int kPanelItems3 = 16;     // A shells of a panel
constexpr int kRecBytes3 = 3072;     // record buffer of a warp (k_moments3)
constexpr int kMomSlots3 = 28;       // moments summed at a time (registers)
// k_transform3 (<= 168 registers): one CTA of 12 warps per SM, whose slab holds the larger
// blocks in fewer element groups than two CTAs of 6 warps would (777 elements of a
// 32-function basis: FP64 500 against 577 us, FP32 484 against 527 with FP64 exponentials).
// Shared memory: geometry and slab.
constexpr int kTrThreads3 = 384;
constexpr int kTrSmem3 = 222 * 1024;

// Record of a primitive triple of a class with D moments: the exponent's three
// coefficients (times log2(e) for ex2_neg3) and the moments' factors w mono_m.
__host__ __device__ constexpr int rec_bytes3(int nv) { return (24 + 8 * nv + 15) / 16 * 16; }

// Canonical classes L0 >= L1 >= L2, in the order of class3().
#define AOK_CLASSES3(X) \
    X(0, 0, 0, 1) X(1, 0, 0, 1) X(1, 1, 0, 1) X(1, 1, 1, 1) X(2, 0, 0, 1) X(2, 1, 0, 1) X(2, 1, 1, 1) X(2, 2, 0, 1) \
    X(2, 2, 1, 1) X(2, 2, 2, 3) \
    X(3, 0, 0, 1) X(3, 1, 0, 1) X(3, 1, 1, 1) X(3, 2, 0, 1) X(3, 2, 1, 2) X(3, 2, 2, 5) X(3, 3, 0, 2) X(3, 3, 1, 5) \
    X(3, 3, 2, 10) X(3, 3, 3, 10)
// index of a class in the list above; the last column is its number of transform parts
__host__ __device__ constexpr int class3(int l0, int l1, int l2) {
    return l0 * (l0 + 1) * (l0 + 2) / 6 + l1 * (l1 + 1) / 2 + l2;
}
static_assert(class3(2, 2, 2) == 9 && class3(3, 0, 0) == 10 && class3(3, 3, 3) == 19, "class order");
// Moments and recursions are FP64 in both precisions.  With FP32 sums (runs of 8 triples
// folded with TwoSum) and FP32 recursions up to d, p-p-p, d-p-p, d-d-p and d-d-d were off by up
// to 1.3 times as much as with E tables (norm of the block, d-d-p of two primitives per shell:
// 1.03e-7 against 8.2e-8); so they are off by 3e-8 to 4.7e-8 in every class.  777 elements
// take 428 us (490 so), 1,500 take 754 (757), 1,682 of a basis of up to 8 primitives in every
// shell 976 (955).  Up to d FP32 takes its exponentials from ex2 (rounding of the result
// apart, the error that is left); with FP64 ones every class is at 2.5e-8 to 3.6e-8, but 777
// elements cost another 40 us and 1,500 another 65.  Blocks with an f shell have them in
// FP64, as their E tables do.
template <typename FT>
__host__ __device__ constexpr bool fast_exp3(int l0) { return sizeof(FT) == 4 && l0 <= 2; }
struct ClassInfo3 {
    short D, ops, parts, comps;
};
#define AOK_X(a, b, c, np) {(short)Prog3<a, b, c, 0, 1>::D, (short)Prog3<a, b, c, 0, 1>::NOPS, np, ncart(a) * ncart(b) * ncart(c)},
constexpr ClassInfo3 kClass3Host[20] = {AOK_CLASSES3(AOK_X)};
static __constant__ ClassInfo3 kClass3[20] = {AOK_CLASSES3(AOK_X)};
#undef AOK_X

// Canonical order of a shell triple: o[k] = the role (0: A, 1: B, 2: C) of centre k.
struct Canon3 {
    int o0, o1, o2, cls;
};
__host__ __device__ constexpr Canon3 canon3(int la, int lb, int lc) {
    Canon3 r{0, 1, 2, 0};
    int l0 = la, l1 = lb, l2 = lc;
    if (l0 < l1) {
        const int t = l0, u = r.o0;
        l0 = l1;
        l1 = t;
        r.o0 = r.o1;
        r.o1 = u;
    }
    if (l1 < l2) {
        const int t = l1, u = r.o1;
        l1 = l2;
        l2 = t;
        r.o1 = r.o2;
        r.o2 = u;
    }
    if (l0 < l1) {
        const int t = l0, u = r.o0;
        l0 = l1;
        l1 = t;
        r.o0 = r.o1;
        r.o1 = u;
    }
    r.cls = class3(l0, l1, l2);
    return r;
}

struct Panel3 {
    short sa0, nsa, sb, sc;  // A shells [sa0, sa0 + nsa)
    int comps;               // slab elements of a batch element: sum of NA NB NC
    short passes, pass;      // the slab holds 32 / passes elements: this panel's are those of pass
    int tab, nout;           // the panel's output elements: entries [tab, tab + nout) of the table
    int moff;                // first moment
};
// One block (shell triple) for the moment kernel.
struct Item3 {
    short sa, sb, sc, cls;
    int moff;                // first moment
};
// Output element of a panel: the slab elements that the aliased layout adds into it (at
// most 2 x 2; the rest name the row's zero element, index comps) and its offset from the panel's first element.
struct __align__(16) Out3 {
    short o[4];
    int at, pad;
};

// Tile geometry in shared memory, one column per lane: A - B, A - C, B - C.
template <typename FT>
struct __align__(16) Geo3 {
    long long at[32];  // the element's first output
    double d[9][32];
};

// Slab elements (of FT) that a CTA has.
template <typename FT>
__host__ __device__ constexpr int slab_room3() {
    return (kTrSmem3 - 2 * (int)sizeof(Geo3<FT>)) / (int)sizeof(FT);
}

// The pair differences A - B, A - C, B - C in FP64 (exact for FP32 positions); positions
// are multiplied by s when use_s (the orbital path's lengthscale).
template <typename FT>
__device__ __forceinline__ void differences3(double (&d)[9], const FT* A, const FT* B, const FT* C, FT s, bool use_s) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        FT a = A[c], b = B[c], cc = C[c];
        if (use_s) {
            a *= s;
            b *= s;
            cc *= s;
        }
        d[c] = (double)a - (double)b;
        d[3 + c] = (double)a - (double)cc;
        d[6 + c] = (double)b - (double)cc;
    }
}

// index of centre pair (p, q)
__device__ __forceinline__ int pair3(int p, int q) { return p + q - 1; }

// A block's inputs for one unit, canonical centre order.
template <typename FT>
struct Block3 {
    const FT* z[3];
    const FT* c[3];
    int n[3];
    int o0, o1, o2;
};

// --------------------------------------------------------------------------
// Phase 1: moments
// --------------------------------------------------------------------------

// Factors of the moment slots K0 + J from the powers of w r0 (w in front), r1, r2 and h.
template <int L0, int L1, int L2, int K0>
struct Slots3 {
    using PR = Prog3<L0, L1, L2, 0, 1>;
    static constexpr typename PR::Mono kMono = PR::monos();
    template <int J>
    static __device__ __forceinline__ double one(const double* pa, const double* pb, const double* pg,
                                                 const double* ph) {
        constexpr int a = kMono.a[K0 + J], b = kMono.b[K0 + J], g = kMono.g[K0 + J], d = kMono.d[K0 + J];
        return (pa[a] * pb[b]) * (pg[g] * ph[d]);
    }
    template <int... J>
    static __device__ __forceinline__ void fill(double* v, const double* pa, const double* pb, const double* pg,
                                                const double* ph, Seq<J...>) {
        ((v[J] = one<J>(pa, pb, pg, ph)), ...);
    }
};

// Record of the triple (a, b, c) with coefficients ca, cb, cc: moment slots [K0, K0 + NV)
// of the class.
template <int L0, int L1, int L2, int K0, int NV, bool EX2>
__device__ __forceinline__ void fill_rec3(char* rec, double ca, double cb, double cc, double a, double b, double c) {
    using PR = Prog3<L0, L1, L2, 0, 1>;
    const double q = a + b + c, iq = 1.0 / q, x = 3.14159265358979323846 * iq;
    double* k = reinterpret_cast<double*>(rec);
    const double l2e = EX2 ? 1.4426950408889634074 : 1.0;
    k[0] = a * b * iq * l2e;
    k[1] = a * c * iq * l2e;
    k[2] = b * c * iq * l2e;
    double pa[PR::MA], pb[PR::MB], pg[PR::MG], ph[PR::n / 2 + 1];
    pa[0] = ca * cb * cc * (x * sqrt(x));
    pb[0] = pg[0] = ph[0] = 1.0;
#pragma unroll
    for (int i = 1; i < PR::MA; ++i) pa[i] = pa[i - 1] * (a * iq);
#pragma unroll
    for (int i = 1; i < PR::MB; ++i) pb[i] = pb[i - 1] * (b * iq);
#pragma unroll
    for (int i = 1; i < PR::MG; ++i) pg[i] = pg[i - 1] * (c * iq);
#pragma unroll
    for (int i = 1; i <= PR::n / 2; ++i) ph[i] = ph[i - 1] * (0.5 * iq);
    Slots3<L0, L1, L2, K0>::fill(k + 3, pa, pb, pg, ph, MakeSeq<NV>{});
}

// 2^-x with x given in FP64 (log2 units): the integer part goes into the exponent field,
// the fraction (|f| <= 1/2, so one rounding to FP32 costs 2^-26 of the result) through
// ex2.  x is cut off at 200 through its high word, and 2^-n is 0 from n = 127 on; an
// infinite or NaN distance is put back by the caller.
__device__ __forceinline__ float ex2_neg3(double x) {
    const double magic = 6755399441055744.0;  // 1.5 * 2^52: the sum's low word is round(x)
    x = __hiloint2double(min(__double2hiint(x), 0x40690000), __double2loint(x));
    const double t = x + magic;
    const float f = __double2float_rn(x - (t - magic));
    return ex2_approx(-f) * __int_as_float(min(max(127 - __double2loint(t), 0), 255) << 23);
}
// e^{-arg} of one record for the lane's squared distances.
template <bool EX2>
__device__ __forceinline__ double rec_exp3(const char* rec, double R0, double R1, double R2) {
    const double2 k = *reinterpret_cast<const double2*>(rec);
    const double k2 = *reinterpret_cast<const double*>(rec + 16);
    if (EX2) return (double)ex2_neg3(fma(k2, R2, fma(k.y, R1, k.x * R0)));
    return exp(-fma(k2, R2, fma(k.y, R1, k.x * R0)));
}
// Adds e times one record's factors.
template <int NV>
__device__ __forceinline__ void add_rec3(const char* rec, double e, double (&part)[NV]) {
    part[0] = fma(e, *reinterpret_cast<const double*>(rec + 24), part[0]);
#pragma unroll
    for (int i = 1; i < NV; i += 2) {
        const double2 w = *reinterpret_cast<const double2*>(rec + 24 + 8 * i);
        part[i] = fma(e, w.x, part[i]);
        if (i + 1 < NV) part[i + 1] = fma(e, w.y, part[i + 1]);
    }
}

// Moment slots [K0, K0 + NV) of a block's triples [q0, q1): the warp builds records batch
// by batch in its buffer (one per lane) and every lane sums them for its element.
template <int L0, int L1, int L2, int K0, int NV, typename FT>
__device__ __forceinline__ void moments3(const Block3<FT>& bl, int q0, int q1, char* buf, const double (&R)[3],
                                         double (&sum)[NV]) {
    const int lane = threadIdx.x & 31;
    constexpr int RB = rec_bytes3(NV);
    constexpr bool EX2 = fast_exp3<FT>(L0);
    constexpr int NB = kRecBytes3 / RB >= 32 ? 32 : kRecBytes3 / RB;
    static_assert(NB >= 8, "record buffer");
    const int n12 = bl.n[1] * bl.n[2], n2 = bl.n[2];
    const float f12 = 1.f / (float)n12, f2 = 1.f / (float)n2;
    const double R0 = R[pair3(bl.o0, bl.o1)], R1 = R[pair3(bl.o0, bl.o2)], R2 = R[pair3(bl.o1, bl.o2)];
#pragma unroll
    for (int i = 0; i < NV; ++i) sum[i] = 0.0;
#pragma unroll 1
    for (int qb = q0; qb < q1; qb += NB) {
        const int m = min(NB, q1 - qb);
        __syncwarp();
        if (lane < m) {
            // (i, j, k) of triple q; the quotients by FP32 estimate, put right by at most one
            const int q = qb + lane;
            int i = (int)((float)q * f12), r = q - i * n12;
            i += r >= n12 ? 1 : r < 0 ? -1 : 0;
            r = q - i * n12;
            int j = (int)((float)r * f2), k = r - j * n2;
            j += k >= n2 ? 1 : k < 0 ? -1 : 0;
            k = r - j * n2;
            fill_rec3<L0, L1, L2, K0, NV, EX2>(buf + lane * RB, (double)bl.c[0][i], (double)bl.c[1][j],
                                               (double)bl.c[2][k], (double)bl.z[0][i], (double)bl.z[1][j],
                                               (double)bl.z[2][k]);
        }
        __syncwarp();
        int q = 0;
        const char* rec = buf;
        // the exponentials of kIlp triples in flight, then their multiply-adds
        constexpr int kIlp = NV <= 6 ? 4 : 2;
#pragma unroll 1
        for (; q + kIlp <= m; q += kIlp, rec += kIlp * RB) {
            double e[kIlp];
#pragma unroll
            for (int u = 0; u < kIlp; ++u) e[u] = rec_exp3<EX2>(rec + u * RB, R0, R1, R2);
#pragma unroll
            for (int u = 0; u < kIlp; ++u) add_rec3<NV>(rec + u * RB, e[u], sum);
        }
#pragma unroll 1
        for (; q < m; ++q, rec += RB) add_rec3<NV>(rec, rec_exp3<EX2>(rec, R0, R1, R2), sum);
    }
}

// The slots from K0 on, kMomSlots3 at a time, to row out[32 (slot)] (a column per lane).
// split: the CTA's warps take a share of the triples each and their sums meet in xbuf, added
// in warp order by warp 0.
template <int L0, int L1, int L2, int K0, typename FT>
__device__ __forceinline__ void moments3_from(const Block3<FT>& bl, int n, char* buf, const double (&R)[3], double* out,
                                              bool split, double* xbuf) {
    constexpr int D = Prog3<L0, L1, L2, 0, 1>::D, NCH = (D + kMomSlots3 - 1) / kMomSlots3, S = (D + NCH - 1) / NCH;
    constexpr int NV = K0 + S <= D ? S : D - K0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int per = split ? (n + 8 * kWarps3 - 1) / (8 * kWarps3) * 8 : n;
    const int q0 = split ? min(n, warp * per) : 0, q1 = min(n, q0 + per);
    double sum[NV];
    moments3<L0, L1, L2, K0, NV, FT>(bl, q0, q1, buf, R, sum);
    if (split) {
        if (warp > 0) {
#pragma unroll
            for (int i = 0; i < NV; ++i) xbuf[((warp - 1) * kMomSlots3 + i) * 32 + lane] = sum[i];
        }
        __syncthreads();
        if (warp == 0) {
#pragma unroll 1
            for (int w = 0; w < kWarps3 - 1; ++w)
#pragma unroll
                for (int i = 0; i < NV; ++i) sum[i] += xbuf[(w * kMomSlots3 + i) * 32 + lane];
        }
        __syncthreads();  // xbuf is free for the next slots
    }
    if (!split || warp == 0) {
        if constexpr (fast_exp3<FT>(L0)) {  // NaN when a distance is infinite or NaN (see ex2_neg3)
            const double all = R[0] + R[1] + R[2], bad = all - all;
#pragma unroll
            for (int i = 0; i < NV; ++i) sum[i] += bad;
        }
#pragma unroll
        for (int i = 0; i < NV; ++i) out[32 * (K0 + i) + lane] = sum[i];
    }
    if constexpr (K0 + S < D) moments3_from<L0, L1, L2, K0 + S, FT>(bl, n, buf, R, out, split, xbuf);
}
template <int L0, int L1, int L2, typename FT>
__device__ __noinline__ void moments3_call(const Block3<FT>& bl, int n, char* buf, const double (&R)[3], double* out,
                                           bool split, double* xbuf) {
    moments3_from<L0, L1, L2, 0, FT>(bl, n, buf, R, out, split, xbuf);
}

// --------------------------------------------------------------------------
// A block: its components into the slab row of the lane's element
// --------------------------------------------------------------------------
template <typename FT>
struct Dest3 {
    FT* row;         // the block's first component
    int t0, t1, t2;  // strides of the canonical centres' components
    bool on;         // the lane's element is in this pass
};
template <int L0, int L1, int L2, int PART, int NP, typename FT>
__device__ __forceinline__ void transform3_slab(const double* mom, const Geo3<FT>& g, int o0, int o1, int o2,
                                                const Dest3<FT>& to) {
    const int lane = threadIdx.x & 31;
    const double* m = mom + lane;
    double d01[3], d02[3], d12[3];
    if constexpr (L0 > 0) {
        const double s01 = o0 < o1 ? 1.0 : -1.0, s02 = o0 < o2 ? 1.0 : -1.0, s12 = o1 < o2 ? 1.0 : -1.0;
        const int p01 = 3 * pair3(o0, o1), p02 = 3 * pair3(o0, o2), p12 = 3 * pair3(o1, o2);
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            d01[x] = s01 * g.d[p01 + x][lane];
            d02[x] = s02 * g.d[p02 + x][lane];
            d12[x] = s12 * g.d[p12 + x][lane];
        }
    }
    FT* row = to.row;
    const int t0 = to.t0, t1 = to.t1, t2 = to.t2;
    const bool on = to.on;
    transform3<L0, L1, L2, PART, NP, double>([&](int k) { return __ldcs(m + 32 * k); }, d01, d02, d12,
                                             [&](int c0, int c1, int c2, double v) {
                                                 if (on) row[c0 * t0 + c1 * t1 + c2 * t2] = (FT)v;
                                             });
}
template <int L0, int L1, int L2, int PART, int NP, typename FT>
__device__ __noinline__ void transform3_call(const double* mom, const Geo3<FT>& g, int o0, int o1, int o2,
                                             const Dest3<FT>& to) {
    transform3_slab<L0, L1, L2, PART, NP, FT>(mom, g, o0, o1, o2, to);
}

template <int L0, int L1, int L2, int NP, typename FT>
__device__ __forceinline__ void block3_part(int part, const double* mom, const Geo3<FT>& g, int o0, int o1, int o2,
                                            const Dest3<FT>& to) {
    if constexpr (L0 + L1 + L2 <= 2) {
        transform3_slab<L0, L1, L2, 0, 1, FT>(mom, g, o0, o1, o2, to);
    } else {
        switch (part) {
            case 0: if constexpr (NP > 0) transform3_call<L0, L1, L2, 0, NP, FT>(mom, g, o0, o1, o2, to); break;
            case 1: if constexpr (NP > 1) transform3_call<L0, L1, L2, 1, NP, FT>(mom, g, o0, o1, o2, to); break;
            case 2: if constexpr (NP > 2) transform3_call<L0, L1, L2, 2, NP, FT>(mom, g, o0, o1, o2, to); break;
            case 3: if constexpr (NP > 3) transform3_call<L0, L1, L2, 3, NP, FT>(mom, g, o0, o1, o2, to); break;
            case 4: if constexpr (NP > 4) transform3_call<L0, L1, L2, 4, NP, FT>(mom, g, o0, o1, o2, to); break;
            case 5: if constexpr (NP > 5) transform3_call<L0, L1, L2, 5, NP, FT>(mom, g, o0, o1, o2, to); break;
            case 6: if constexpr (NP > 6) transform3_call<L0, L1, L2, 6, NP, FT>(mom, g, o0, o1, o2, to); break;
            case 7: if constexpr (NP > 7) transform3_call<L0, L1, L2, 7, NP, FT>(mom, g, o0, o1, o2, to); break;
            case 8: if constexpr (NP > 8) transform3_call<L0, L1, L2, 8, NP, FT>(mom, g, o0, o1, o2, to); break;
            case 9: if constexpr (NP > 9) transform3_call<L0, L1, L2, 9, NP, FT>(mom, g, o0, o1, o2, to); break;
            default: break;
        }
        static_assert(NP <= 10, "transform parts");
    }
}

// --------------------------------------------------------------------------
// Kernel
// --------------------------------------------------------------------------
template <typename FT>
struct Ov3Params {
    FT* out;
    const FT* posA;
    const FT* posB;
    const FT* posC;
    const FT* pz;        // compact primitive lists: zeta, coef of (species g, shell s) at (g ns + s) K
    const FT* pc;
    const int* pn;       // their lengths, (g ns + s)
    const int* perm;
    const int4* tiles;
    const int* ntiles;
    unsigned* counter;   // [0] the moment kernel's, [1] the transform kernel's
    const Item3* items;  // every block in queue order (k_prepm3)
    const int* segs;     // segment starts in items (nseg + 1 entries); nseg, H, pick at segs[nitems + 1], [nitems + 2], [nitems + 3]
    const Panel3* panels;
    const Out3* table;   // the panels' output elements
    double* mom;         // moments of tile t: mom + (t - tile0) * slots * 32
    int tile0, round;    // this launch's tiles: [tile0, tile0 + round)
    int nitems, npanels, slots, ns, K, N, NZ;
    FT scale;
    int use_scale;
    int boff[kMaxShells + 1];
    signed char l[kMaxShells];
};

// Work unit = (segment, W tiles): a run of consecutive items of the queue order for W
// consecutive tiles, one tile per warp.  The first H segments (heavy single items) take one
// tile per unit instead, their triples shared out over the W warps.  A CTA claims one unit
// at a time from one counter, segment-major, so the warps of a CTA run the same routines.
template <typename FT>
__global__ void __launch_bounds__(kThreads3, kMomCtas3) k_moments3(const __grid_constant__ Ov3Params<FT> P) {
    constexpr int W = kWarps3;
    __shared__ __align__(16) char recbuf[W][kRecBytes3];
    __shared__ __align__(16) double xbuf[(W - 1) * kMomSlots3 * 32];
    __shared__ unsigned claim;
    pdl_wait();  // launched programmatically after k_overlap3c or the last round: the bins, the prep's order and the
                 // buffers are complete past here
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (!P.segs[P.nitems + 3]) return;  // explicit tables
    const int ntiles = min(*P.ntiles - P.tile0, P.round), nseg = P.segs[P.nitems + 1], H = P.segs[P.nitems + 2];
    if (ntiles <= 0) return;
    const unsigned ngroups = (unsigned)(ntiles + W - 1) / W;
    const unsigned nsplit = (unsigned)H * (unsigned)ntiles, total = nsplit + ngroups * (unsigned)(nseg - H);
    for (;;) {
        if (threadIdx.x == 0) claim = atomicAdd(P.counter, 1u);
        __syncthreads();
        const unsigned u = claim;
        __syncthreads();
        if (u >= total) break;
        const bool split = u < nsplit;
        int sg, tile;
        if (split) {
            sg = (int)(u / (unsigned)ntiles);
            tile = (int)(u % (unsigned)ntiles);
        } else {
            sg = H + (int)((u - nsplit) / ngroups);
            tile = (int)((u - nsplit) % ngroups) * W + warp;
            if (tile >= ntiles) continue;
        }
        const int4 td = P.tiles[P.tile0 + tile];
        const int b = P.perm[td.y + (lane < td.z ? lane : 0)];
        double d[9], R[3];
        differences3(d, P.posA + 3 * (size_t)b, P.posB + 3 * (size_t)b, P.posC + 3 * (size_t)b, P.scale,
                     P.use_scale != 0);
#pragma unroll
        for (int i = 0; i < 3; ++i) R[i] = fma(d[3 * i + 2], d[3 * i + 2], fma(d[3 * i + 1], d[3 * i + 1], d[3 * i] * d[3 * i]));
        // the tile's species triple (key ((ga NZ) + gb) NZ + gc; 0 on the single-species path)
        const int ga = td.x / (P.NZ * P.NZ), gb = (td.x / P.NZ) % P.NZ, gc = td.x % P.NZ;
        const int i0 = P.segs[sg], i1 = P.segs[sg + 1];
#pragma unroll 1
        for (int it = i0; it < i1; ++it) {
            const Item3 wi = P.items[it];
            const Canon3 cn = canon3(P.l[wi.sa], P.l[wi.sb], P.l[wi.sc]);
            Block3<FT> bl;
            bl.o0 = cn.o0;
            bl.o1 = cn.o1;
            bl.o2 = cn.o2;
            const int o[3] = {cn.o0, cn.o1, cn.o2};
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const int sh = o[k] == 0 ? ga * P.ns + wi.sa : o[k] == 1 ? gb * P.ns + wi.sb : gc * P.ns + wi.sc;
                bl.z[k] = P.pz + (size_t)sh * P.K;
                bl.c[k] = P.pc + (size_t)sh * P.K;
                bl.n[k] = P.pn[sh];
            }
            const int n = bl.n[0] * bl.n[1] * bl.n[2];
            if (n == 0) continue;  // k_transform3 writes zeros
            double* out = P.mom + ((size_t)tile * P.slots + wi.moff) * 32;
            switch (wi.cls) {
#define AOK_X(a, b, c, np)                                                           \
    case class3(a, b, c):                                                            \
        if constexpr (a + b + c <= 2)                                                \
            moments3_from<a, b, c, 0, FT>(bl, n, recbuf[warp], R, out, split, xbuf); \
        else                                                                         \
            moments3_call<a, b, c, FT>(bl, n, recbuf[warp], R, out, split, xbuf);    \
        break;
                AOK_CLASSES3(AOK_X)
                default: break;
#undef AOK_X
            }
        }
    }
}

// A unit's panel, tile and tasks, in shared memory.
struct Unit3 {
    Panel3 pn;
    int tile, cnt;                // tile (-1: no unit), its elements
    int t[kPanelItems3 + 1];      // first task of each block
    int zero[kPanelItems3];       // a shell is absent from its species
    int soff[kPanelItems3], moff[kPanelItems3];  // first slab element, first moment row
};

template <typename FT>
__global__ void __launch_bounds__(kTrThreads3, 1) k_transform3(const __grid_constant__ Ov3Params<FT> P) {
    extern __shared__ __align__(16) char smem[];
    __shared__ Unit3 units[2];
    __shared__ unsigned s_u[2];
    __shared__ int count;
    pdl_wait();  // launched programmatically after the moment kernel
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    Geo3<FT>* geo = reinterpret_cast<Geo3<FT>*>(smem);
    FT* slab = reinterpret_cast<FT*>(smem + 2 * sizeof(Geo3<FT>));
    if (!P.segs[P.nitems + 3]) return;  // explicit tables
    const int left = min(*P.ntiles - P.tile0, P.round);
    if (left <= 0) return;
    const unsigned ntiles = (unsigned)left, total = (unsigned)P.npanels * ntiles;
    const size_t N2 = (size_t)P.N * P.N;
    // one warp: the unit u = (panel, tile), its geometry, blocks and tasks into slot f
    auto fetch = [&](int f, unsigned u) {
        Unit3& U = units[f];
        if (u >= total) {
            if (lane == 0) U.tile = -1;
            return;
        }
        const int tile = (int)(u % ntiles);
        const int4 td = P.tiles[P.tile0 + tile];
        const Panel3 pn = P.panels[u / ntiles];
        const int b = P.perm[td.y + (lane < td.z ? lane : 0)];
        const int key = td.x, ga = key / (P.NZ * P.NZ), gb = (key / P.NZ) % P.NZ, gc = key % P.NZ;
        const bool on = lane < pn.nsa;
        const int sa = pn.sa0 + (on ? lane : 0), la = P.l[sa], lb = P.l[pn.sb], lc = P.l[pn.sc];
        const ClassInfo3 ci = kClass3[canon3(la, lb, lc).cls];
        const bool zero = P.pn[ga * P.ns + sa] * P.pn[gb * P.ns + pn.sb] * P.pn[gc * P.ns + pn.sc] == 0;
        const int t0 = on ? (zero ? 1 : ci.parts) : 0, s0 = on ? ncart(la) * ncart(lb) * ncart(lc) : 0, m0 = on ? ci.D : 0;
        int t = t0, so = s0, m = m0;
#pragma unroll
        for (int o = 1; o < kPanelItems3; o <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, t, o), y = __shfl_up_sync(0xffffffffu, so, o),
                      z = __shfl_up_sync(0xffffffffu, m, o);
            if (lane >= o) {
                t += x;
                so += y;
                m += z;
            }
        }
        if (on) {
            U.t[lane] = t - t0;
            U.zero[lane] = zero;
            U.soff[lane] = so - s0;
            U.moff[lane] = pn.moff + m - m0;
        }
        if (lane == pn.nsa - 1) U.t[pn.nsa] = t;
        if (lane == 0) {
            U.pn = pn;
            U.tile = tile;
            U.cnt = td.z;
        }
        geo[f].at[lane] = (long long)b * (long long)(N2 * P.N);
        double d[9];
        differences3(d, P.posA + 3 * (size_t)b, P.posB + 3 * (size_t)b, P.posC + 3 * (size_t)b, P.scale,
                     P.use_scale != 0);
#pragma unroll
        for (int i = 0; i < 9; ++i) geo[f].d[i][lane] = d[i];
    };
    if (warp == 0) {
        unsigned u = 0;
        if (lane == 0) u = atomicAdd(P.counter + 1, 1u);
        fetch(0, __shfl_sync(0xffffffffu, u, 0));
    }
    int f = 0;
    for (;;) {
        if (threadIdx.x == 0) count = 0;
        __syncthreads();  // the unit is set up, the slab is free
        const Unit3& U = units[f];
        if (U.tile < 0) break;
        if (threadIdx.x == kTrThreads3 - 1) s_u[f] = atomicAdd(P.counter + 1, 1u);  // the next unit
        const Panel3 pn = U.pn;
        const int lb = P.l[pn.sb], lc = P.l[pn.sc], NB = ncart(lb), NC = ncart(lc);
        const int lanes = 32 / pn.passes, rowlen = (pn.comps + 1) | 1;
        const int nt = pn.pass * lanes < U.cnt ? U.t[pn.nsa] : 0;  // a partial tile may not reach this pass
        const double* tile_mom = P.mom + (size_t)U.tile * P.slots * 32;
        FT* row = slab + (size_t)(lane & (lanes - 1)) * rowlen;
        if (warp == 0 && lane < lanes) row[pn.comps] = FT(0);
        for (;;) {
            int t = 0;
            if (lane == 0) t = atomicAdd(&count, 1);
            t = nt - 1 - __shfl_sync(0xffffffffu, t, 0);  // the highest momenta first
            if (t < 0) break;
            int i = pn.nsa - 1;
            while (t < U.t[i]) --i;
            const int part = t - U.t[i], la = P.l[pn.sa0 + i], NA = ncart(la);
            Dest3<FT> to;
            to.on = lane / lanes == pn.pass;
            to.row = row + U.soff[i];
            if (U.zero[i]) {
                if (to.on)
                    for (int k = 0; k < NA * NB * NC; ++k) to.row[k] = FT(0);
                continue;
            }
            const Canon3 cn = canon3(la, lb, lc);
            const int sj = NA, sk = NA * NB;
            to.t0 = cn.o0 == 0 ? 1 : cn.o0 == 1 ? sj : sk;
            to.t1 = cn.o1 == 0 ? 1 : cn.o1 == 1 ? sj : sk;
            to.t2 = cn.o2 == 0 ? 1 : cn.o2 == 1 ? sj : sk;
            const double* mom = tile_mom + (size_t)U.moff[i] * 32;
            switch (cn.cls) {
#define AOK_X(a, b, c, np) \
    case class3(a, b, c): block3_part<a, b, c, np, FT>(part, mom, geo[f], cn.o0, cn.o1, cn.o2, to); break;
                AOK_CLASSES3(AOK_X)
                default: break;
#undef AOK_X
            }
        }
        __syncthreads();
        if (warp == kTrThreads3 / 32 - 1) fetch(f ^ 1, s_u[f]);
        // the slab streams out
        const int e0 = pn.pass * lanes, ne = min(lanes, U.cnt - e0);
        FT* out = P.out + (size_t)P.boff[pn.sc] * N2 + (size_t)P.boff[pn.sb] * P.N + P.boff[pn.sa0];
        const long long* at = geo[f].at + e0;
#pragma unroll 1
        for (int x0 = 32 * warp; x0 < pn.nout; x0 += kTrThreads3) {
            const int x = x0 + lane;
            const bool in = x < pn.nout;
            const Out3 q = P.table[pn.tab + (in ? x : 0)];
            const bool two = __any_sync(0xffffffffu, q.o[1] != pn.comps),
                       four = __any_sync(0xffffffffu, q.o[2] != pn.comps);
            if (!in) continue;
            FT* o = out + q.at;
            const FT* r = slab + q.o[0];
            if (!two) {
#pragma unroll 8
                for (int e = 0; e < ne; ++e, r += rowlen) __stcs(o + at[e], *r);
            } else if (!four) {
                const FT* r1 = slab + q.o[1];
#pragma unroll 8
                for (int e = 0; e < ne; ++e, r += rowlen, r1 += rowlen) __stcs(o + at[e], *r + *r1);
            } else {
                r = slab;
#pragma unroll 4
                for (int e = 0; e < ne; ++e, r += rowlen)
                    __stcs(o + at[e], ((r[q.o[0]] + r[q.o[1]]) + r[q.o[2]]) + r[q.o[3]]);
            }
        }
        f ^= 1;
    }
}

// Takes the local memory of the transform's routines from the device (1.6 GB of stack over
// all SMs, which the driver keeps), through a launch that finds the tables picked and
// returns: *e says whether there was room.
template <typename FT>
inline int reserve_moments3(aok_plan* p, cudaError_t* e) {
    Ov3Params<FT> P;
    memset(&P, 0, sizeof(P));
    P.segs = p->d_segsm;
    P.nitems = p->nitemsm;
    auto tr = k_transform3<FT>;
    const int st = kernel_prepare((const void*)tr, kTrSmem3, kTrThreads3, nullptr);
    if (st != AOK_OK) return st;
    *e = cudaMemsetAsync(p->d_segsm + p->nitemsm + 3, 0, sizeof(int), p->side);
    if (*e == cudaSuccess) *e = launch_pdl(tr, dim3(p->num_sms), dim3(kTrThreads3), kTrSmem3, p->side, P);
    if (*e == cudaSuccess) *e = cudaStreamSynchronize(p->side);
    return AOK_OK;
}

template <typename FT>
inline int launch_moments3(aok_plan* p, void* out, const void* posA, const void* posB, const void* posC, int64_t B,
                           double lengthscale, cudaStream_t s) {
    Ov3Params<FT> P;
    memset(&P, 0, sizeof(P));
    P.out = (FT*)out;
    P.posA = (const FT*)posA;
    P.posB = (const FT*)posB;
    P.posC = (const FT*)posC;
    P.pz = (const FT*)p->d_pp3;
    P.pc = (const FT*)p->d_pp3 + p->ns * p->K * p->NZ;
    P.pn = p->d_npp3;
    P.perm = p->d_perm;
    P.tiles = p->d_tiles;
    P.ntiles = p->d_ntiles;
    P.items = (const Item3*)p->d_orderm;
    P.segs = p->d_segsm;
    P.panels = (const Panel3*)p->d_panels3;
    P.table = (const Out3*)p->d_out3;
    P.mom = (double*)p->d_mom3;
    P.round = p->round3;
    P.nitems = p->nitemsm;
    P.npanels = p->npanels3;
    P.slots = p->slots3;
    P.ns = (int)p->ns;
    P.K = (int)p->K;
    P.N = (int)p->N;
    P.NZ = (int)p->NZ;
    P.scale = (FT)lengthscale;
    P.use_scale = (FT)lengthscale != FT(1);
    for (int i = 0; i <= p->ns; ++i) P.boff[i] = (int)p->boff[i];
    for (int i = 0; i < p->ns; ++i) P.l[i] = (signed char)p->ls[i];
    auto mom = k_moments3<FT>;
    auto tr = k_transform3<FT>;
    int st;
    if ((st = kernel_prepare((const void*)mom, 0, kThreads3, nullptr)) != AOK_OK) return st;
    if ((st = kernel_prepare((const void*)tr, kTrSmem3, kTrThreads3, nullptr)) != AOK_OK) return st;
    // a tile per 32 elements and one partial tile per species triple
    const int64_t most = (B + 31) / 32 + p->NZ * p->NZ * p->NZ;
    const int rounds = (int)((most + p->round3 - 1) / p->round3);
    cudaError_t e = cudaSuccess;
    for (int r = 0; r < rounds && e == cudaSuccess; ++r) {
        P.tile0 = r * p->round3;
        P.counter = p->d_cnt3 + 2 * r;
        e = launch_pdl(mom, dim3(p->num_sms * kMomCtas3), dim3(kThreads3), 0, s, P);
        if (e == cudaSuccess) e = launch_pdl(tr, dim3(p->num_sms), dim3(kTrThreads3), kTrSmem3, s, P);
    }
    timing_end(p, s);  // begun before the explicit tables' kernel (launch_ov3)
    return cuda_status(e, "k_transform3");
}

}  // namespace m3
}  // namespace aok
