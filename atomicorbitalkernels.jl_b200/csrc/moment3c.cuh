// moment3c.cuh -- 3-center overlap by primitive-triple moments (early contraction).
//
// For one shell triple on centres P0, P1, P2 (momenta L0 >= L1 >= L2, the caller
// permutes its centres into this order) a primitive triple (a, b, c) enters the
// Obara-Saika recursion of its overlap only through
//   r0 = a/q, r1 = b/q, r2 = c/q, h = 1/2q   (q = a + b + c),
// because the Gaussian product centre Q satisfies
//   Q - P0 = -(r1 d01 + r2 d02),  Q - P1 = r0 d01 - r2 d12,  Q - P2 = r0 d02 + r1 d12
// with d01 = P0 - P1 and so on.  Every component of the block is therefore a
// polynomial in the geometry times monomials r0^al r1^be r2^ga h^de of one degree
// al + be + ga + 2 de = L0 + L1 + L2, and the sum over primitive triples is taken
// first:
//   M_m = sum over triples of w e^{-arg} mono_m        (D moments: 1 s-s-s, 41 d-d-d)
// The recursion then runs once per block on vectors of moments,
//   [n + 1_i]_m = (Q - P_s)_i o [n]_m + sum_t n_t,i [n - 1_i of centre t]_{m + h},
// where multiplying by r_s raises a moment index.  Centre 0 is built up first, then
// 1, then 2.  Only the (node, moment) values that a wanted component needs are
// formed: d-d-d takes 3,210 multiply-adds for 216 components, against 1,100 for every
// primitive triple with explicit E tables.
//
// Prog3 lists these operations at compile time, depth first in the order of the
// components (a value is formed right before its first use, so that few are alive at a
// time; in f-f-f, f-f-d and f-d-d still more than the registers hold).  NP > 1 splits the
// components by centre 0's component into NP programs.
#pragma once

#include <utility>

#include "aok_common.cuh"

namespace aok {

template <int... I>
using Seq = std::integer_sequence<int, I...>;
template <int N>
using MakeSeq = std::make_integer_sequence<int, N>;

// Cartesian sub-components of a shell: all (x, y, z) with x + y + z <= L, indexed by
// degree, then in the component order of aok_common.cuh.
__host__ __device__ constexpr int nsub(int L) { return (L + 1) * (L + 2) * (L + 3) / 6; }
__host__ __device__ constexpr int sub_index(int x, int y, int z) {
    const int d = x + y + z, n = y + z;
    return d * (d + 1) * (d + 2) / 6 + n * (n + 1) / 2 + z;
}

struct Op3 {
    short dst;            // value slot written
    short q1, q2;         // moment-raised predecessors (Q - P_s: first and second ratio)
    short h[3];           // h-raised lower neighbours, or -1
    signed char c[3];     // their integer factors
    signed char s, ax;    // raised centre and axis
    short out;            // packed component c0 + 16 c1 + 256 c2 when dst is a block component, else -1
};

template <int L0, int L1, int L2, int PART, int NP>
struct Prog3 {
    static constexpr int n = L0 + L1 + L2;
    static constexpr int S0 = nsub(L0), S1 = nsub(L1), S2 = nsub(L2), NN = S0 * S1 * S2;
    static constexpr int NC0 = ncart(L0), NC1 = ncart(L1), NC2 = ncart(L2);
    static constexpr int C0 = PART * NC0 / NP, C1 = (PART + 1) * NC0 / NP;  // this part's components of centre 0
    // moments by (al, be, ga): al <= L1 + L2 and so on bounds each exponent; de follows
    static constexpr int MA = L1 + L2 + 1, MB = L0 + L2 + 1, MG = L0 + L1 + 1;
    static constexpr int MM = MA * MB * MG;
    static constexpr int WORDS = (MM + 63) / 64;
    struct Sub {
        signed char x, y, z;
    };
    struct State {
        unsigned long long need[NN][WORDS] = {};
        unsigned long long done[NN][WORDS] = {};
        short base[NN] = {};
        Sub sub[20] = {};
        int nslots = 0, D = 0, nops = 0;
    };
    static constexpr int midx(int a, int b, int g) { return (g * MB + b) * MA + a; }
    static constexpr int node(int i0, int i1, int i2) { return (i0 * S1 + i1) * S2 + i2; }
    struct Raise {
        int s, ax, parent;
        int low[3], c[3];
    };
    static constexpr int subi(const Sub& u, int ax, int d) {
        return sub_index(u.x + (ax == 0 ? d : 0), u.y + (ax == 1 ? d : 0), u.z + (ax == 2 ? d : 0));
    }
    static constexpr int comp(const Sub& u, int ax) { return ax == 0 ? u.x : ax == 1 ? u.y : u.z; }
    static constexpr void fill_sub(State& st) {
        for (int d = 0; d <= 3; ++d)
            for (int c = 0; c < ncart(d); ++c) {
                const int x = cart_x(d, c), y = cart_y(d, c), z = cart_z(d, c);
                st.sub[sub_index(x, y, z)] = Sub{(signed char)x, (signed char)y, (signed char)z};
            }
    }
    // how node (i0, i1, i2) is raised: the last centre that has quanta, its first axis
    static constexpr Raise raise(const State& st, int i0, int i1, int i2) {
        Raise r{};
        int id[3] = {i0, i1, i2};
        r.s = i2 ? 2 : i1 ? 1 : 0;
        const Sub u = st.sub[id[r.s]];
        r.ax = u.x ? 0 : u.y ? 1 : 2;
        id[r.s] = subi(u, r.ax, -1);
        r.parent = node(id[0], id[1], id[2]);
        for (int t = 0; t < 3; ++t) {
            const int q = comp(st.sub[id[t]], r.ax);
            r.c[t] = q;
            r.low[t] = -1;
            if (q) {
                int lo[3] = {id[0], id[1], id[2]};
                lo[t] = subi(st.sub[id[t]], r.ax, -1);
                r.low[t] = node(lo[0], lo[1], lo[2]);
            }
        }
        return r;
    }
    static constexpr bool get(const unsigned long long (&w)[WORDS], int m) { return (w[m >> 6] >> (m & 63)) & 1ull; }
    static constexpr void set(unsigned long long (&w)[WORDS], int m) { w[m >> 6] |= 1ull << (m & 63); }
    static constexpr int slot(const State& st, int nd, int m) {
        int k = st.base[nd];
        for (int w = 0; w < (m >> 6); ++w) k += popc(st.need[nd][w]);
        return k + popc(st.need[nd][m >> 6] & ((1ull << (m & 63)) - 1ull));
    }
    static constexpr int popc(unsigned long long v) {
        int c = 0;
        for (; v; v &= v - 1) ++c;
        return c;
    }
    // ratio raised by Q - P_s: first and second term
    static constexpr int q1of(int s) { return s == 0 ? midx(0, 1, 0) : midx(1, 0, 0); }
    static constexpr int q2of(int s) { return s == 2 ? midx(0, 1, 0) : midx(0, 0, 1); }

    static constexpr State analyse() {
        State st{};
        fill_sub(st);
        const int b0 = nsub(L0) - NC0, b1 = nsub(L1) - NC1, b2 = nsub(L2) - NC2;
        for (int a = C0; a < C1; ++a)
            for (int b = 0; b < NC1; ++b)
                for (int c = 0; c < NC2; ++c) set(st.need[node(b0 + a, b1 + b, b2 + c)], 0);
        // parents and lower neighbours have smaller sub-indices of the raised centre or of another
        // one, never larger: a descending sweep sees every need before the node is expanded
        for (int i2 = S2 - 1; i2 >= 0; --i2)
            for (int i1 = S1 - 1; i1 >= 0; --i1)
                for (int i0 = S0 - 1; i0 >= 0; --i0) {
                    const int nd = node(i0, i1, i2);
                    if (nd == 0) continue;
                    bool any = false;
                    for (int w = 0; w < WORDS; ++w) any = any || st.need[nd][w] != 0;
                    if (!any) continue;
                    const Raise r = raise(st, i0, i1, i2);
                    for (int w = 0; w < WORDS; ++w)
                        for (unsigned long long v = st.need[nd][w]; v; v &= v - 1) {
                            const int m = 64 * w + popc((v & (0ull - v)) - 1ull);
                            set(st.need[r.parent], m + q1of(r.s));
                            set(st.need[r.parent], m + q2of(r.s));
                            for (int t = 0; t < 3; ++t)
                                if (r.low[t] >= 0) set(st.need[r.low[t]], m);  // h: same (al, be, ga)
                            ++st.nops;
                        }
                }
        int k = 0;
        for (int nd = 0; nd < NN; ++nd) {
            st.base[nd] = (short)k;
            for (int w = 0; w < WORDS; ++w) k += popc(st.need[nd][w]);
            if (nd == 0) st.D = k;
        }
        st.nslots = k;
        return st;
    }
    static constexpr State kState = analyse();
    static constexpr int D = kState.D, NSLOT = kState.nslots, NOPS = kState.nops;

    // this part's moment slots among the whole block's (Prog3<..., 0, 1>)
    struct Map {
        short at[D > 0 ? D : 1];
    };
    static constexpr Map map_moments() {
        using Whole = Prog3<L0, L1, L2, 0, 1>;
        Map o{};
        int k = 0;
        for (int m = 0; m < MM; ++m)
            if (get(kState.need[0], m)) o.at[k++] = (short)Whole::slot(Whole::kState, 0, m);
        return o;
    }
    // the exponents of moment slot k (node 0's needed monomials in index order)
    struct Mono {
        signed char a[D > 0 ? D : 1], b[D > 0 ? D : 1], g[D > 0 ? D : 1], d[D > 0 ? D : 1];
    };
    static constexpr Mono monos() {
        Mono o{};
        int k = 0;
        for (int m = 0; m < MM; ++m)
            if (get(kState.need[0], m)) {
                const int a = m % MA, b = (m / MA) % MB, g = m / (MA * MB);
                o.a[k] = (signed char)a;
                o.b[k] = (signed char)b;
                o.g[k] = (signed char)g;
                o.d[k] = (signed char)((n - a - b - g) / 2);
                ++k;
            }
        return o;
    }
    struct Ops {
        Op3 op[NOPS > 0 ? NOPS : 1];
        int n;
    };
    static constexpr void emit(State& st, Ops& o, int i0, int i1, int i2, int m, int out) {
        const int nd = node(i0, i1, i2);
        if (nd == 0 || get(st.done[nd], m)) return;
        set(st.done[nd], m);
        const Raise r = raise(st, i0, i1, i2);
        const int p0 = r.parent / (S1 * S2), p1 = r.parent / S2 % S1, p2 = r.parent % S2;
        emit(st, o, p0, p1, p2, m + q1of(r.s), -1);
        emit(st, o, p0, p1, p2, m + q2of(r.s), -1);
        Op3 e{};
        for (int t = 0; t < 3; ++t) {
            e.h[t] = -1;
            e.c[t] = (signed char)r.c[t];
            if (r.low[t] >= 0) {
                emit(st, o, r.low[t] / (S1 * S2), r.low[t] / S2 % S1, r.low[t] % S2, m, -1);
                e.h[t] = (short)slot(st, r.low[t], m);
            }
        }
        e.dst = (short)slot(st, nd, m);
        e.q1 = (short)slot(st, r.parent, m + q1of(r.s));
        e.q2 = (short)slot(st, r.parent, m + q2of(r.s));
        e.s = (signed char)r.s;
        e.ax = (signed char)r.ax;
        e.out = (short)out;
        o.op[o.n++] = e;
    }
    static constexpr Ops make() {
        Ops o{};
        State st = kState;
        const int b0 = nsub(L0) - NC0, b1 = nsub(L1) - NC1, b2 = nsub(L2) - NC2;
        for (int a = C0; a < C1; ++a)
            for (int b = 0; b < NC1; ++b)
                for (int c = 0; c < NC2; ++c) emit(st, o, b0 + a, b1 + b, b2 + c, 0, a + 16 * b + 256 * c);
        return o;
    }
};

// Each operation is its own template instance, so that every index is a constant and the
// values live in registers.
template <int L0, int L1, int L2, int PART, int NP, typename FT>
struct Run3 {
    using PR = Prog3<L0, L1, L2, PART, NP>;
    static constexpr typename PR::Ops kOps = PR::make();
    static constexpr typename PR::Map kMap = PR::map_moments();

    template <int I, typename Sink>
    static __host__ __device__ __forceinline__ void step(FT* v, const FT* d01, const FT* d02, const FT* d12,
                                                         Sink& sink) {
        if constexpr (I < PR::NOPS) {
            constexpr Op3 e = kOps.op[I];
            constexpr int ax = e.ax, q1 = e.q1, q2 = e.q2, h0 = e.h[0], h1 = e.h[1], h2 = e.h[2], dst = e.dst;
            constexpr FT k0 = FT(e.c[0]), k1 = FT(e.c[1]), k2 = FT(e.c[2]);
            FT t;
            if constexpr (e.s == 0)
                t = -fma(d01[ax], v[q1], d02[ax] * v[q2]);
            else if constexpr (e.s == 1)
                t = fma(d01[ax], v[q1], -(d12[ax] * v[q2]));
            else
                t = fma(d02[ax], v[q1], d12[ax] * v[q2]);
            if constexpr (h0 >= 0) t = fma(k0, v[h0], t);
            if constexpr (h1 >= 0) t = fma(k1, v[h1], t);
            if constexpr (h2 >= 0) t = fma(k2, v[h2], t);
            v[dst] = t;
            if constexpr (e.out >= 0) {
                constexpr int c0 = e.out & 15, c1 = (e.out >> 4) & 15, c2 = e.out >> 8;
                sink(c0, c1, c2, t);
            }
        }
    }
    template <int I0, typename Sink, int... I>
    static __host__ __device__ __forceinline__ void steps(FT* v, const FT* d01, const FT* d02, const FT* d12,
                                                          Sink& sink, Seq<I...>) {
        (step<I0 + I>(v, d01, d02, d12, sink), ...);
    }
    template <typename Sink, int... B>
    static __host__ __device__ __forceinline__ void blocks(FT* v, const FT* d01, const FT* d02, const FT* d12,
                                                           Sink& sink, Seq<B...>) {
        (steps<64 * B>(v, d01, d02, d12, sink, MakeSeq<64>{}), ...);
    }
    template <int K, typename Load>
    static __host__ __device__ __forceinline__ FT load_one(Load& ld) {
        constexpr int at = kMap.at[K];
        return ld(at);
    }
    template <typename Load, int... K>
    static __host__ __device__ __forceinline__ void load(FT* v, Load& ld, Seq<K...>) {
        ((v[K] = load_one<K>(ld)), ...);
    }
};

// Runs the program on the block's moments: ld(k) gives moment k (in the slot order of the
// whole block's monos()), sink(c0, c1, c2, value) takes every component of the part.
// d01, d02, d12: the centre differences.
template <int L0, int L1, int L2, int PART, int NP, typename FT, typename Load, typename Sink>
__host__ __device__ __forceinline__ void transform3(Load&& ld, const FT (&d01)[3], const FT (&d02)[3],
                                                    const FT (&d12)[3], Sink&& sink) {
    using R = Run3<L0, L1, L2, PART, NP, FT>;
    using PR = typename R::PR;
    FT v[PR::NSLOT];
    R::load(v, ld, MakeSeq<PR::D>{});
    if constexpr (PR::n == 0)
        sink(0, 0, 0, v[0]);
    else
        R::blocks(v, d01, d02, d12, sink, MakeSeq<(PR::NOPS + 63) / 64>{});
}

}  // namespace aok
