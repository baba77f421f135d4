// overlap3c_kernel.cuh -- batched 3-center overlap kernel, templated on the
// element type (instantiated in overlap3c_f32.cu / overlap3c_f64.cu).
//
// Replaces batch_V_kernel! (src/integrals/kernels_3c.jl:12-162):
//   V_{mu nu lambda}(b) = int phi_mu(r - A_b) phi_nu(r - B_b) phi_lambda(r - C_b) dr.
// Per primitive triple the three Gaussians combine at Q = (aA + bB + cC)/q
// with prefactor c_a c_b c_c (pi/q)^{3/2} exp(-(ab|AB|^2 + ac|AC|^2 + bc|BC|^2)/q)
// (the reference's mu|AB|^2 + nu|PC|^2), and the 1-D factors are the t = 0
// three-index coefficients, built with the Obara-Saika form
//   E[i+1][j][k] = QA E + (i E[i-1][j][k] + j E[i][j-1][k] + k E[i][j][k-1]) / 2q
// and its j / k analogues (QB, QC); QA = -(b AB + c AC)/q, QB = (a AB - c BC)/q,
// QC = (a AC + b BC)/q are formed directly.  The reference's aliased layout
// lin = c1 + (2la+1) c2 + (2la+1)(2lb+1) c3 (kernels_3c.jl:146-160) is
// reproduced at compile time.
//
// Execution: tiles of 32 batch elements (lane = element); shell-triple classes
// (la, lb, lc <= 2) compile-time specialised (classes with an f shell:
// run_item3_f, below).  Items are whole shell-triple blocks or chunks of whole
// output pages; (segment, tile) units, a segment being a run of items of about
// equal cost, are drained from one global queue, heaviest first (k_overlap3c
// below).
#pragma once

#include <algorithm>
#include <cstring>

#include "aok_internal.h"

namespace aok {

constexpr int kMaxL3 = 3;        // shells up to f
constexpr int kMaxL3Spec = 2;    // compile-time specialised classes up to d
constexpr int kClsF3 = 100;      // Item3 class code of a triple with an f shell: kClsF3 + la*16 + lb*4 + lc
constexpr int kThreads3 = 128;
constexpr int kSplitM3 = 9;  // largest block that the CTA's warps may share (heavy items, l_a + l_b + l_c <= 2)
// Claims per CTA (a segment for the CTA's W tiles, heavy items shared out over
// its warps) in FP32; claims per warp of (item, tile) units in FP64, whose
// longer and more variable exponentials balance better in small units (both
// measured on config 4).
template <typename FT> constexpr bool kCtaClaims3 = sizeof(FT) == 4;
constexpr int kShortM3 = 18;  // FP32C blocks of >= this many elements take a plain path when n <= 8

__host__ __device__ constexpr int pages_per_chunk3(int la, int lb) {
    return (ncart(la) * ncart(lb)) >= 36 ? 1 : 36 / (ncart(la) * ncart(lb));
}
__host__ __device__ constexpr int nchunks3(int la, int lb, int lc) {
    return (ncart(lc) + pages_per_chunk3(la, lb) - 1) / pages_per_chunk3(la, lb);
}

// Geometry-free primitive-triple record (FP64-computed).  FP32: the exponent
// coefficients k_xy = (x y / q) log2(e) stay FP64, so that the exponent
// k_ab |AB|^2 + k_ac |AC|^2 + k_bc |BC|^2 is three FP64 FMAs split into hi + lo
// floats for ex2; the rest is FP32.
struct __align__(16) PTf {
    double kab, kac, kbc;
    float w, ra, rb, rc, oo2q, pad;
};
struct __align__(16) PTd {
    double w, kab, kac, kbc, ra, rb, rc, oo2q;
};
template <typename FT> struct PTT;
template <> struct PTT<float> { using type = PTf; };
template <> struct PTT<double> { using type = PTd; };

struct Item3 {
    int16_t cls;    // la*9 + lb*3 + lc, or kClsF3 + la*16 + lb*4 + lc with an f shell
    int16_t chunk;
    int16_t sa, sb, sc, pad;
};


template <typename FT> struct Geo3;
template <> struct Geo3<float> {
    float AB[3], AC[3], BC[3];
    double R2[3];  // |AB|^2, |AC|^2, |BC|^2 of the FP32 positions, in FP64
};
template <> struct Geo3<double> {
    double AB[3], AC[3], BC[3];
    double R2[3];
};

// Positions multiplied by s when use_s (the orbital path's lengthscale), then
// the pair differences; FP32: the differences of the FP32 values exact in FP64.
__device__ __forceinline__ void load_geo3(Geo3<float>& g, const float* A, const float* B, const float* C, float s,
                                          bool use_s) {
    double r[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        float a = A[c], b = B[c], cc = C[c];
        if (use_s) {
            a *= s;
            b *= s;
            cc *= s;
        }
        const double ab = (double)a - (double)b, ac = (double)a - (double)cc,
                     bc = (double)b - (double)cc;  // exact differences of FP32 values
        g.AB[c] = (float)ab;
        g.AC[c] = (float)ac;
        g.BC[c] = (float)bc;
        r[0] += ab * ab;
        r[1] += ac * ac;
        r[2] += bc * bc;
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) g.R2[i] = r[i];
}
__device__ __forceinline__ void load_geo3(Geo3<double>& g, const double* A, const double* B, const double* C,
                                          double s, bool use_s) {
#pragma unroll
    for (int i = 0; i < 3; ++i) g.R2[i] = 0.0;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        double a = A[c], b = B[c], cc = C[c];
        if (use_s) {
            a *= s;
            b *= s;
            cc *= s;
        }
        g.AB[c] = a - b;
        g.AC[c] = a - cc;
        g.BC[c] = b - cc;
        g.R2[0] += g.AB[c] * g.AB[c];
        g.R2[1] += g.AC[c] * g.AC[c];
        g.R2[2] += g.BC[c] * g.BC[c];
    }
}

// E[i][j][k] for i <= LA, j <= LB, k <= LC, seeded with E[0][0][0] = e000.
template <int LA, int LB, int LC, typename FT>
__device__ __forceinline__ void build_E3(FT (&E)[LA + 1][LB + 1][LC + 1], FT QA, FT QB, FT QC, FT o2q, FT e000) {
    E[0][0][0] = e000;
#pragma unroll
    for (int k = 0; k <= LC; ++k)
#pragma unroll
        for (int j = 0; j <= LB; ++j)
#pragma unroll
            for (int i = 0; i <= LA; ++i) {
                if (i == 0 && j == 0 && k == 0) continue;
                // raise the first non-zero index from its predecessor
                FT v;
                if (k > 0 && i == 0 && j == 0) {
                    v = QC * E[0][0][k - 1];
                    if (k >= 2) v += (FT(k - 1) * o2q) * E[0][0][k - 2];
                } else if (i == 0) {
                    v = QB * E[0][j - 1][k];
                    FT c = FT(0);
                    if (j >= 2) c += FT(j - 1) * E[0][j - 2][k];
                    if (k >= 1) c += FT(k) * E[0][j - 1][k - 1];
                    v += o2q * c;
                } else {
                    v = QA * E[i - 1][j][k];
                    FT c = FT(0);
                    if (i >= 2) c += FT(i - 1) * E[i - 2][j][k];
                    if (j >= 1) c += FT(j) * E[i - 1][j - 1][k];
                    if (k >= 1) c += FT(k) * E[i - 1][j][k - 1];
                    v += o2q * c;
                }
                E[i][j][k] = v;
            }
}

template <int LA, int LB, int LC>
struct Class3 {
    static constexpr int NA = ncart(LA), NB = ncart(LB), NC = ncart(LC);
    static constexpr int PS = NA * NB;            // elements per output page of the block
    static constexpr int NE = PS * NC;
    static constexpr int N1 = 2 * LA + 1, N2 = 2 * LB + 1;
    static constexpr int PPC = pages_per_chunk3(LA, LB);
};

// Record of one primitive triple, FP64-computed (the product's weight, the
// exponent coefficients, the exponent ratios and 1/2q).
__device__ __forceinline__ void fill_pt(PTf& r, double ca, double cb, double cc, double a, double b, double c) {
    const double q = a + b + c, iq = 1.0 / q, x = 3.14159265358979323846 * iq, l2e = 1.4426950408889634074;
    r.w = (float)(ca * cb * cc * (x * sqrt(x)));
    r.kab = a * b * iq * l2e;
    r.kac = a * c * iq * l2e;
    r.kbc = b * c * iq * l2e;
    r.ra = (float)(a * iq);
    r.rb = (float)(b * iq);
    r.rc = (float)(c * iq);
    r.oo2q = (float)(0.5 * iq);
    r.pad = 0.f;
}
__device__ __forceinline__ void fill_pt(PTd& r, double ca, double cb, double cc, double a, double b, double c) {
    const double q = a + b + c, iq = 1.0 / q, x = 3.14159265358979323846 * iq;
    r.w = ca * cb * cc * (x * sqrt(x));
    r.kab = a * b * iq;
    r.kac = a * c * iq;
    r.kbc = b * c * iq;
    r.ra = a * iq;
    r.rb = b * iq;
    r.rc = c * iq;
    r.oo2q = 0.5 * iq;
}

// The three shells' primitives for one work unit (the tile's species): the
// compact lists of non-zero (zeta, coef) slots (k_prep3c) and their lengths.
template <typename FT>
struct Prim3 {
    const FT* z[3];
    const FT* c[3];
    int n[3];
};

// Records q0 .. q0 + 31 of the unit into the warp's buffer, one per lane (FP64
// arithmetic), in (ip, jp, kp) order; the caller brackets it with __syncwarp.
template <typename PT, typename FT>
__device__ __forceinline__ void gen_records3(PT* buf, const Prim3<FT>& pr, int q0, int n, int lane) {
    const int q = q0 + lane;
    if (q >= n) return;
    const int nb = pr.n[1], nc = pr.n[2];
    const int ip = q / (nb * nc), jp = (q / nc) % nb, kp = q % nc;
    fill_pt(buf[lane], (double)pr.c[0][ip], (double)pr.c[1][jp], (double)pr.c[2][kp], (double)pr.z[0][ip],
            (double)pr.z[1][jp], (double)pr.z[2][kp]);
}

// One primitive triple's products E_x E_y E_z added into the sums of the
// chunk's block elements [L0, L0 + M) (aliased lin order).
template <int LA, int LB, int LC, int L0, int M, typename FT>
__device__ __forceinline__ void add_products3(FT ra, FT rb, FT rc, FT o2q, FT e000, const Geo3<FT>& g,
                                              FT (&part)[M]) {
    using CI = Class3<LA, LB, LC>;
    FT Ex[LA + 1][LB + 1][LC + 1], Ey[LA + 1][LB + 1][LC + 1], Ez[LA + 1][LB + 1][LC + 1];
    build_E3<LA, LB, LC, FT>(Ex, -(rb * g.AB[0] + rc * g.AC[0]), ra * g.AB[0] - rc * g.BC[0],
                             ra * g.AC[0] + rb * g.BC[0], o2q, e000);
    build_E3<LA, LB, LC, FT>(Ey, -(rb * g.AB[1] + rc * g.AC[1]), ra * g.AB[1] - rc * g.BC[1],
                             ra * g.AC[1] + rb * g.BC[1], o2q, FT(1));
    build_E3<LA, LB, LC, FT>(Ez, -(rb * g.AB[2] + rc * g.AC[2]), ra * g.AB[2] - rc * g.BC[2],
                             ra * g.AC[2] + rb * g.BC[2], o2q, FT(1));
#pragma unroll
    for (int c3 = 0; c3 < CI::NC; ++c3)
#pragma unroll
        for (int c2 = 0; c2 < CI::NB; ++c2)
#pragma unroll
            for (int c1 = 0; c1 < CI::NA; ++c1) {
                const int lin = c1 + CI::N1 * c2 + CI::N1 * CI::N2 * c3;
                if (lin >= L0 && lin < L0 + M) {
                    const FT yz = Ey[cart_y(LA, c1)][cart_y(LB, c2)][cart_y(LC, c3)] *
                                  Ez[cart_z(LA, c1)][cart_z(LB, c2)][cart_z(LC, c3)];
                    part[lin - L0] = fma(Ex[cart_x(LA, c1)][cart_x(LB, c2)][cart_x(LC, c3)], yz, part[lin - L0]);
                }
            }
}

// FP32: 2^-x with x = k_ab |AB|^2 + k_ac |AC|^2 + k_bc |BC|^2 (log2 units) in FP64,
// split into hi + lo floats; FP64: exp(-x).
template <int LA, int LB, int LC, int L0, int M>
__device__ __forceinline__ void add_rec3(const PTf& r, const Geo3<float>& g, float (&part)[M]) {
    const double x = fma(r.kbc, g.R2[2], fma(r.kac, g.R2[1], r.kab * g.R2[0]));
    const float xh = __double2float_rn(x), xl = __double2float_rn(x - (double)xh);
    const float e000 = (ex2_approx(-xh) * fmaf(-0.6931471805599453f, xl, 1.f)) * r.w;
    add_products3<LA, LB, LC, L0, M, float>(r.ra, r.rb, r.rc, r.oo2q, e000, g, part);
}
template <int LA, int LB, int LC, int L0, int M>
__device__ __forceinline__ void add_rec3(const PTd& r, const Geo3<double>& g, double (&part)[M]) {
    const double e000 = exp(-(r.kab * g.R2[0] + r.kac * g.R2[1] + r.kbc * g.R2[2])) * r.w;
    add_products3<LA, LB, LC, L0, M, double>(r.ra, r.rb, r.rc, r.oo2q, e000, g, part);
}

// Classes with l_a + l_b + l_c <= 2 take two triples per loop step (two
// independent exponential chains in flight); larger classes one.
template <int LA, int LB, int LC>
__host__ __device__ constexpr bool pair_step3() {
    return LA + LB + LC <= 2;
}

// lin (0-based, within the block) -> offset in the output;
// block element (i, j, k) = (lin % NA, (lin / NA) % NB, lin / PS).
// With split, the CTA's warps share one tile: warp w takes the record chunks
// w, w + W, ... and the partial sums meet in xbuf (blocks of <= kSplitM3).
template <int LA, int LB, int LC, int C>
__device__ __forceinline__ void run_item3(const Prim3<float> pr, PTf* buf, const Geo3<float> g, float* dst, int N,
                                       bool split, void* xbuf, bool valid) {
    const int lane = threadIdx.x & 31, n = pr.n[0] * pr.n[1] * pr.n[2];
    using CI = Class3<LA, LB, LC>;
    constexpr int P0 = C * CI::PPC, P1 = (C + 1) * CI::PPC < CI::NC ? (C + 1) * CI::PPC : CI::NC;
    constexpr int L0 = P0 * CI::PS, M = (P1 - P0) * CI::PS;
    if constexpr (M >= kShortM3) {
        // Large blocks of at most 8 triples (one run): plain FP32 sums, so that the
        // (hi, lo) registers of the compensated path are not live here.
        if (n <= 8) {
            float part[M];
#pragma unroll
            for (int m = 0; m < M; ++m) part[m] = 0.f;
            __syncwarp();
            gen_records3(buf, pr, 0, n, lane);
            __syncwarp();
#pragma unroll 1
            for (int q = 0; q < n; ++q) add_rec3<LA, LB, LC, L0, M>(buf[q], g, part);
            if (!valid) return;
#pragma unroll
            for (int m = 0; m < M; ++m) {
                const int lin = L0 + m, pg = lin / CI::PS;
                const int i = lin % CI::NA, j = (lin / CI::NA) % CI::NB;
                dst[(size_t)pg * N * N + (size_t)j * N + i] = part[m];
            }
            return;
        }
    }
    // Compensated contraction: runs of up to 8 triples are summed in part[], and
    // each run is folded into hi + lo with TwoSum.
    float hi[M], lo[M], part[M];
#pragma unroll
    for (int m = 0; m < M; ++m) {
        hi[m] = 0.f;
        lo[m] = 0.f;
        part[m] = 0.f;
    }
    const int w = threadIdx.x >> 5, q00 = split ? 32 * w : 0, qs = split ? 32 * (kThreads3 / 32) : 32;
#pragma unroll 1
    for (int q0 = q00; q0 < n; q0 += qs) {
      __syncwarp();
      gen_records3(buf, pr, q0, n, lane);
      __syncwarp();
      const int m = min(32, n - q0);
#pragma unroll 1
      for (int q8 = 0; q8 < m; q8 += 8) {
        if (q0 + q8 > q00) {
#pragma unroll
            for (int k = 0; k < M; ++k) {
                float s, e;
                two_sum(hi[k], part[k], s, e);
                hi[k] = s;
                part[k] = 0.f;
                lo[k] += e;
            }
        }
        const int qe = min(q8 + 8, m);
        int q = q8;
        if constexpr (pair_step3<LA, LB, LC>()) {
#pragma unroll 1
            for (; q + 1 < qe; q += 2) {
                const PTf r0 = buf[q], r1 = buf[q + 1];
                add_rec3<LA, LB, LC, L0, M>(r0, g, part);
                add_rec3<LA, LB, LC, L0, M>(r1, g, part);
            }
        }
#pragma unroll 1
        for (; q < qe; ++q) add_rec3<LA, LB, LC, L0, M>(buf[q], g, part);
      }
    }
    float sum[M];
#pragma unroll
    for (int m = 0; m < M; ++m) {
        float e;
        two_sum(hi[m], part[m], sum[m], e);
        lo[m] += e;
    }
    if constexpr (M <= kSplitM3) {
        if (split) {
            // the other warps' (sum, lo) pairs, added to warp 0's in warp order
            float2* x = reinterpret_cast<float2*>(xbuf);
            if (w > 0) {
#pragma unroll
                for (int m = 0; m < M; ++m) x[((w - 1) * kSplitM3 + m) * 32 + lane] = make_float2(sum[m], lo[m]);
            }
            __syncthreads();
            if (w > 0) return;
#pragma unroll 1
            for (int v = 0; v < kThreads3 / 32 - 1; ++v)
#pragma unroll
                for (int m = 0; m < M; ++m) {
                    const float2 o = x[(v * kSplitM3 + m) * 32 + lane];
                    float s2, e;
                    two_sum(sum[m], o.x, s2, e);
                    sum[m] = s2;
                    lo[m] += o.y + e;
                }
        }
    }
    if (!valid) return;
#pragma unroll
    for (int m = 0; m < M; ++m) {
        const int lin = L0 + m, pg = lin / CI::PS;
        const int i = lin % CI::NA, j = (lin / CI::NA) % CI::NB;
        dst[(size_t)pg * N * N + (size_t)j * N + i] = sum[m] + lo[m];
    }
}

template <int LA, int LB, int LC, int C>
__device__ __forceinline__ void run_item3(const Prim3<double> pr, PTd* buf, const Geo3<double> g, double* dst, int N,
                                       bool split, void* xbuf, bool valid) {
    const int lane = threadIdx.x & 31, n = pr.n[0] * pr.n[1] * pr.n[2];
    using CI = Class3<LA, LB, LC>;
    constexpr int P0 = C * CI::PPC, P1 = (C + 1) * CI::PPC < CI::NC ? (C + 1) * CI::PPC : CI::NC;
    constexpr int L0 = P0 * CI::PS, M = (P1 - P0) * CI::PS;
    double acc[M];
#pragma unroll
    for (int m = 0; m < M; ++m) acc[m] = 0.0;
    const int w = threadIdx.x >> 5, q00 = split ? 32 * w : 0, qs = split ? 32 * (kThreads3 / 32) : 32;
#pragma unroll 1
    for (int q0 = q00; q0 < n; q0 += qs) {
      __syncwarp();
      gen_records3(buf, pr, q0, n, lane);
      __syncwarp();
      const int m = min(32, n - q0);
      int q = 0;
      if constexpr (pair_step3<LA, LB, LC>()) {
#pragma unroll 1
        for (; q + 1 < m; q += 2) {
            const PTd r0 = buf[q], r1 = buf[q + 1];
            add_rec3<LA, LB, LC, L0, M>(r0, g, acc);
            add_rec3<LA, LB, LC, L0, M>(r1, g, acc);
        }
      }
#pragma unroll 1
      for (; q < m; ++q) add_rec3<LA, LB, LC, L0, M>(buf[q], g, acc);
    }
    if constexpr (M <= kSplitM3) {
        if (split) {
            // the other warps' sums, added to warp 0's in warp order
            double* x = reinterpret_cast<double*>(xbuf);
            if (w > 0) {
#pragma unroll
                for (int m = 0; m < M; ++m) x[((w - 1) * kSplitM3 + m) * 32 + lane] = acc[m];
            }
            __syncthreads();
            if (w > 0) return;
#pragma unroll 1
            for (int v = 0; v < kThreads3 / 32 - 1; ++v)
#pragma unroll
                for (int m = 0; m < M; ++m) acc[m] += x[(v * kSplitM3 + m) * 32 + lane];
        }
    }
    if (!valid) return;
#pragma unroll
    for (int m = 0; m < M; ++m) {
        const int lin = L0 + m, pg = lin / CI::PS;
        const int i = lin % CI::NA, j = (lin / CI::NA) % CI::NB;
        dst[(size_t)pg * N * N + (size_t)j * N + i] = acc[m];
    }
}

// Classes with an f shell (la, lb or lc = 3) of bases with few primitives (with
// more: overlap3c_moments.cuh), one routine with run-time loops:
// the E tables of the three axes (4 x 4 x 4 each) and the chunk's <= 100 block
// elements live in local memory, and the recursion runs in FP64 for both
// precisions (an FP32 record's exponent coefficients are FP64 already).  The class and chunk follow the specialised path's conventions
// (aliased lin, pages [P0, P1) of the block).  Only the kernel instantiated
// for bases with f shells calls it, so its local memory is not reserved by
// the others.
__device__ __forceinline__ void e3_axis(double (&E)[4][4][4], int la, int lb, int lc, double QA, double QB, double QC,
                                        double o2q, double e000) {
    for (int k = 0; k <= lc; ++k)
        for (int j = 0; j <= lb; ++j)
            for (int i = 0; i <= la; ++i) {
                double v;
                if (i == 0 && j == 0 && k == 0) {
                    v = e000;
                } else if (i == 0 && j == 0) {
                    v = QC * E[0][0][k - 1];
                    if (k >= 2) v += ((k - 1) * o2q) * E[0][0][k - 2];
                } else if (i == 0) {
                    v = QB * E[0][j - 1][k];
                    double c = 0.0;
                    if (j >= 2) c += (j - 1) * E[0][j - 2][k];
                    if (k >= 1) c += k * E[0][j - 1][k - 1];
                    v += o2q * c;
                } else {
                    v = QA * E[i - 1][j][k];
                    double c = 0.0;
                    if (i >= 2) c += (i - 1) * E[i - 2][j][k];
                    if (j >= 1) c += j * E[i - 1][j - 1][k];
                    if (k >= 1) c += k * E[i - 1][j][k - 1];
                    v += o2q * c;
                }
                E[i][j][k] = v;
            }
}

__device__ __forceinline__ double pt_exponent(const PTf* r, const double (&R2)[3]) {
    return (r->kab * R2[0] + r->kac * R2[1] + r->kbc * R2[2]) * 0.69314718055994530942;  // records carry k log2(e)
}
__device__ __forceinline__ double pt_exponent(const PTd* r, const double (&R2)[3]) {
    return r->kab * R2[0] + r->kac * R2[1] + r->kbc * R2[2];
}

template <typename PT, typename FT>
__device__ __noinline__ void run_item3_f(const Prim3<FT> pr, PT* buf, const Geo3<FT> g, FT* dst, int N, int cls,
                                         int chunk, bool valid) {
    const int lane = threadIdx.x & 31, n = pr.n[0] * pr.n[1] * pr.n[2];
    const int c = cls - kClsF3, la = c >> 4, lb = (c >> 2) & 3, lc = c & 3;
    const int NA = ncart(la), NB = ncart(lb), NC = ncart(lc), PS = NA * NB, N1 = 2 * la + 1, N2 = 2 * lb + 1;
    const int ppc = pages_per_chunk3(la, lb);
    const int P0 = chunk * ppc, P1 = min((chunk + 1) * ppc, NC);
    const int L0 = P0 * PS, M = (P1 - P0) * PS;  // <= 100
    // the component pages c3 whose aliased lin can land in [L0, L0 + M)
    const int span = (NA - 1) + N1 * (NB - 1);
    int c3lo = 0, c3hi = NC;
    while (c3lo < NC && N1 * N2 * c3lo + span < L0) ++c3lo;
    while (c3hi > c3lo && N1 * N2 * (c3hi - 1) >= L0 + M) --c3hi;
    double acc[100];
    for (int m = 0; m < M; ++m) acc[m] = 0.0;
    double AB[3], AC[3], BC[3], R2[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        AB[a] = (double)g.AB[a];
        AC[a] = (double)g.AC[a];
        BC[a] = (double)g.BC[a];
        R2[a] = (double)g.R2[a];
    }
    double E[3][4][4][4];
#pragma unroll 1
    for (int q0 = 0; q0 < n; q0 += 32) {
      __syncwarp();
      gen_records3(buf, pr, q0, n, lane);
      __syncwarp();
      const int m = min(32, n - q0);
#pragma unroll 1
      for (int qq = 0; qq < m; ++qq) {
        const PT* r = buf + qq;
        const double w = (double)r->w, ra = (double)r->ra, rb = (double)r->rb, rc = (double)r->rc,
                     o2q = (double)r->oo2q;
        const double e000 = exp(-pt_exponent(r, R2)) * w;
#pragma unroll
        for (int a = 0; a < 3; ++a)
            e3_axis(E[a], la, lb, lc, -(rb * AB[a] + rc * AC[a]), ra * AB[a] - rc * BC[a], ra * AC[a] + rb * BC[a],
                    o2q, a == 0 ? e000 : 1.0);
        for (int c3 = c3lo; c3 < c3hi; ++c3) {
            const int x3 = cart_x(lc, c3), y3 = cart_y(lc, c3), z3 = cart_z(lc, c3);
            for (int c2 = 0; c2 < NB; ++c2) {
                const int x2 = cart_x(lb, c2), y2 = cart_y(lb, c2), z2 = cart_z(lb, c2);
                for (int c1 = 0; c1 < NA; ++c1) {
                    const int lin = c1 + N1 * c2 + N1 * N2 * c3 - L0;
                    if (lin < 0 || lin >= M) continue;
                    acc[lin] += E[0][cart_x(la, c1)][x2][x3] * (E[1][cart_y(la, c1)][y2][y3] *
                                                                  E[2][cart_z(la, c1)][z2][z3]);
                }
            }
        }
      }
    }
    if (!valid) return;
    for (int m = 0; m < M; ++m) {
        const int lin = L0 + m, pg = lin / PS;
        const int i = lin % NA, j = (lin / NA) % NB;
        dst[(size_t)pg * N * N + (size_t)j * N + i] = (FT)acc[m];
    }
}

template <typename PT, typename FT, int LA, int LB, int LC>
__device__ __forceinline__ void run_chunks3(int chunk, const Prim3<FT>& pp, PT* n, const Geo3<FT>& g, FT* dst, int N,
                                            bool split, void* xbuf, bool valid) {
    constexpr int NCH = nchunks3(LA, LB, LC);
    switch (chunk) {
        case 0: run_item3<LA, LB, LC, 0>(pp, n, g, dst, N, split, xbuf, valid); break;
        case 1: if constexpr (NCH > 1) run_item3<LA, LB, LC, 1>(pp, n, g, dst, N, split, xbuf, valid); break;
        case 2: if constexpr (NCH > 2) run_item3<LA, LB, LC, 2>(pp, n, g, dst, N, split, xbuf, valid); break;
        case 3: if constexpr (NCH > 3) run_item3<LA, LB, LC, 3>(pp, n, g, dst, N, split, xbuf, valid); break;
        case 4: if constexpr (NCH > 4) run_item3<LA, LB, LC, 4>(pp, n, g, dst, N, split, xbuf, valid); break;
        case 5: if constexpr (NCH > 5) run_item3<LA, LB, LC, 5>(pp, n, g, dst, N, split, xbuf, valid); break;
        default: break;
    }
}

// pp: the unit's primitive lists; n: the warp's record buffer
template <typename PT, typename FT, bool F3>
__device__ __forceinline__ void dispatch3(int cls, int chunk, const Prim3<FT>& pp, PT* n, const Geo3<FT>& g, FT* dst,
                                          int N, bool split, void* xbuf, bool valid) {
    if constexpr (F3) {
        if (cls >= kClsF3) {
            run_item3_f<PT, FT>(pp, n, g, dst, N, cls, chunk, valid);
            return;
        }
    }
    switch (cls) {
#define AOK_C3(LA, LB, LC) \
    case (LA) * 9 + (LB) * 3 + (LC): run_chunks3<PT, FT, LA, LB, LC>(chunk, pp, n, g, dst, N, split, xbuf, valid); break;
        AOK_C3(0, 0, 0) AOK_C3(0, 0, 1) AOK_C3(0, 0, 2) AOK_C3(0, 1, 0) AOK_C3(0, 1, 1) AOK_C3(0, 1, 2)
        AOK_C3(0, 2, 0) AOK_C3(0, 2, 1) AOK_C3(0, 2, 2) AOK_C3(1, 0, 0) AOK_C3(1, 0, 1) AOK_C3(1, 0, 2)
        AOK_C3(1, 1, 0) AOK_C3(1, 1, 1) AOK_C3(1, 1, 2) AOK_C3(1, 2, 0) AOK_C3(1, 2, 1) AOK_C3(1, 2, 2)
        AOK_C3(2, 0, 0) AOK_C3(2, 0, 1) AOK_C3(2, 0, 2) AOK_C3(2, 1, 0) AOK_C3(2, 1, 1) AOK_C3(2, 1, 2)
        AOK_C3(2, 2, 0) AOK_C3(2, 2, 1) AOK_C3(2, 2, 2)
#undef AOK_C3
        default: break;
    }
}

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
    unsigned* counter;
    const Item3* items;  // every (shell triple, page chunk) in queue order (k_prep3c)
    const int* segs;     // segment starts in items (nseg + 1 entries); nseg, H at segs[nitems + 1], [nitems + 2]
    int nitems, ns, K, N, NZ;
    FT scale;
    int use_scale;
    int boff[kMaxShells + 1];
    const int* pick;     // bases with f shells: nullptr, or where the prep says that moments are taken
};

// Work unit = (segment, W tiles): a run of consecutive items of the queue order
// (k_prep3c: items of one routine together, heaviest first, cut into segments
// of about equal cost; an item heavier than that is a segment of its own) for
// W consecutive tiles of 32 batch elements, one tile per warp, lane = element.
// The first H segments (heavy single items of small blocks, H from k_prep3c)
// take one tile per unit instead, their records shared out over the W warps,
// so that the heaviest items do not set the kernel's length.  A CTA claims
// one unit at a time from one global counter, segment-major, so the warps of a
// CTA run the same routines and the warps in flight few distinct ones
// (instruction-cache locality), and every tile's heaviest items start first; a
// tile's geometry is loaded once per unit.  A lane writes its element's blocks
// straight to the output: a batch element's (N,N,N) slab is contiguous and the
// whole output is written exactly once.  Three CTAs of four warps per SM
// (<= 168 registers).  FP64 claims per warp instead, with about one item per
// segment (kCtaClaims3).
template <typename FT, bool F3>
__global__ void __launch_bounds__(kThreads3, 3) k_overlap3c(const __grid_constant__ Ov3Params<FT> P) {
    using PT = typename PTT<FT>::type;
    constexpr int W = kThreads3 / 32;
    __shared__ PT recbuf[W][32];                                    // each warp's current 32 records
    __shared__ __align__(16) FT xbuf[(W - 1) * kSplitM3 * 32 * (sizeof(FT) == 4 ? 2 : 1)];  // split partial sums
    __shared__ unsigned claim;
    pdl_wait();  // launched programmatically after the prep: its order and the bins are complete past here
    if constexpr (F3)
        if (P.pick && *P.pick) return;  // through moments (overlap3c_moments.cuh)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ntiles = *P.ntiles, nseg = P.segs[P.nitems + 1], H = P.segs[P.nitems + 2];
    const unsigned ngroups = (unsigned)(ntiles + W - 1) / W;
    const unsigned nsplit = (unsigned)H * (unsigned)ntiles, total = nsplit + ngroups * (unsigned)(nseg - H);
    const size_t N2 = (size_t)P.N * P.N, N3 = N2 * P.N;
    for (;;) {
        bool split = false;
        int sg, tile;
        if constexpr (kCtaClaims3<FT>) {
            // one claim per CTA: its warps take the same segment for W consecutive tiles (or share one)
            if (threadIdx.x == 0) claim = atomicAdd(P.counter, 1u);
            __syncthreads();
            const unsigned u = claim;
            __syncthreads();
            if (u >= total) break;
            split = u < nsplit;
            if (split) {
                sg = (int)(u / (unsigned)ntiles);
                tile = (int)(u % (unsigned)ntiles);
            } else {
                sg = H + (int)((u - nsplit) / ngroups);
                tile = (int)((u - nsplit) % ngroups) * W + warp;
                if (tile >= ntiles) continue;
            }
        } else {
            // one claim per warp: (segment, tile), segment-major
            unsigned u = 0;
            if (lane == 0) u = atomicAdd(P.counter, 1u);
            u = __shfl_sync(0xffffffffu, u, 0);
            if (u >= (unsigned)ntiles * (unsigned)nseg) break;
            sg = (int)(u / (unsigned)ntiles);
            tile = (int)(u % (unsigned)ntiles);
        }
        const int4 td = P.tiles[tile];
        const bool valid = lane < td.z;
        const int b = P.perm[td.y + (valid ? lane : 0)];
        Geo3<FT> g;
        load_geo3(g, P.posA + 3 * (size_t)b, P.posB + 3 * (size_t)b, P.posC + 3 * (size_t)b, P.scale,
                  P.use_scale != 0);
        // the tile's species triple (key ((ga NZ) + gb) NZ + gc; 0 on the single-species path)
        const int ga = td.x / (P.NZ * P.NZ), gb = (td.x / P.NZ) % P.NZ, gc = td.x % P.NZ;
        const FT* zA = P.pz + (size_t)ga * P.ns * P.K;
        const FT* cA = P.pc + (size_t)ga * P.ns * P.K;
        const FT* zB = P.pz + (size_t)gb * P.ns * P.K;
        const FT* cB = P.pc + (size_t)gb * P.ns * P.K;
        const FT* zC = P.pz + (size_t)gc * P.ns * P.K;
        const FT* cC = P.pc + (size_t)gc * P.ns * P.K;
        FT* base = P.out + (size_t)b * N3;
        const int i0 = P.segs[sg], i1 = P.segs[sg + 1];
#pragma unroll 1
        for (int it = i0; it < i1; ++it) {
            const Item3 wi = P.items[it];
            Prim3<FT> pr;
            pr.z[0] = zA + (size_t)wi.sa * P.K;
            pr.c[0] = cA + (size_t)wi.sa * P.K;
            pr.n[0] = __ldg(P.pn + ga * P.ns + wi.sa);
            pr.z[1] = zB + (size_t)wi.sb * P.K;
            pr.c[1] = cB + (size_t)wi.sb * P.K;
            pr.n[1] = __ldg(P.pn + gb * P.ns + wi.sb);
            pr.z[2] = zC + (size_t)wi.sc * P.K;
            pr.c[2] = cC + (size_t)wi.sc * P.K;
            pr.n[2] = __ldg(P.pn + gc * P.ns + wi.sc);
            FT* dst = base + (size_t)P.boff[wi.sc] * N2 + (size_t)P.boff[wi.sb] * P.N + P.boff[wi.sa];
            dispatch3<PT, FT, F3>(wi.cls, wi.chunk, pr, recbuf[warp], g, dst, P.N, split, xbuf, valid);
        }
    }
}

template <typename FT, bool F3>
inline int launch_ov3(aok_plan* p, void* out, const void* posA, const void* posB, const void* posC, double lengthscale,
                      cudaStream_t s, bool pdl) {
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
    P.counter = p->d_counter;
    P.items = (const Item3*)p->d_order3;
    P.segs = p->d_segs3;
    P.nitems = p->nitems3;
    P.ns = (int)p->ns;
    P.K = (int)p->K;
    P.N = (int)p->N;
    P.NZ = (int)p->NZ;
    P.scale = (FT)lengthscale;
    P.use_scale = (FT)lengthscale != FT(1);
    for (int i = 0; i <= p->ns; ++i) P.boff[i] = (int)p->boff[i];
    P.pick = p->d_panels3 ? p->d_segsm + p->nitemsm + 3 : nullptr;
    auto kern = k_overlap3c<FT, F3>;
    int occ = 0;
    const int st = kernel_prepare((const void*)kern, 0, kThreads3, &occ);
    if (st != AOK_OK) return st;
    timing_begin(p, s);
    cudaError_t e;
    // timing events recorded around the kernel sit between it and the prep: launch it plainly then
    const bool timed = !p->ev.empty() && 2 * p->ev_used + 1 < (int)p->ev.size();
    if (pdl && !timed) {
        e = launch_pdl(kern, dim3(p->num_sms * std::max(occ, 1)), dim3(kThreads3), 0, s, P);
    } else {
        kern<<<p->num_sms * std::max(occ, 1), kThreads3, 0, s>>>(P);
        e = cudaGetLastError();
    }
    if (!P.pick) timing_end(p, s);  // else after the moment path's kernels
    return cuda_status(e, "k_overlap3c");
}

}  // namespace aok
