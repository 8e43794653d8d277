// Device hashers of the Merkle path: Poseidon, Poseidon2, Monolith
// (Goldilocks, width 12), Poseidon-BN128 and Keccak-256 over Goldilocks words,
// each one thread per hash with the whole state in registers; Poseidon also
// on six and on two threads per hash, Poseidon2 also on six and Poseidon-BN128
// on five (end of file), for latency-bound work.
//
// Semantics follow zeknox:
//   Poseidon   native/poseidon/poseidon.cu:602-791 (4 full, 22 partial,
//              4 full rounds; x^7; MDS circulant + diag(8,0..0))
//   Poseidon2  native/poseidon2/poseidon2.cu:61-209
//   Keccak     native/keccak/keccak.cu:42-135 (rate 136 B, 0x01 .. 0x80 pad,
//              digest word 3 masked to its low byte)
//   Monolith   native/monolith/monolith.cu:117-233
//   Poseidon-BN128  native/poseidon/poseidon_bn128.cu:111-193
//   sponge     native/poseidon/poseidon_permutation.cuh:226-276 (rate 8,
//              overwrite mode, n <= 4 copies and zero-pads)
#pragma once
#include <stdint.h>

#include <type_traits>

#include "gl64.cuh"
#include "zk_constants.h"

namespace zk {

// ---------------------------------------------------- exact FP64 layers
// The linear layers with small integer coefficients run on the FP64 pipe, next
// to the integer pipes that carry the S-box products: each lane is split into
// its two 32-bit halves, each half-vector goes through the layer in doubles,
// and every product and partial sum is an integer below 2^53 in magnitude, so
// the FP64 arithmetic is exact.
//
// No conversion instruction is used: the 64-bit pattern of a non-negative
// integer n < 2^53 read as a double is n 2^-1074 (a denormal, and from 2^52 on
// the first normals), so integers go in as the word pair (x, 0) and results
// come out as their own bit pattern.  FP64 runs at the same rate on denormals
// (63.5 DFMA per clock and SM measured either way).
//
// Cost model behind the splits below (measured on the Poseidon leaf kernel): a
// scheduler slot per instruction, two for an FP64 instruction and two for a
// 32 x 32 -> 64-bit multiply; that kernel runs at 90 % of it (FP64 matrix
// instructions take 11-12 slots next to integer work, for what is 8 FP64
// instructions' worth of products, a quarter of them padding).
__host__ __device__ constexpr uint64_t cx_canon(uint64_t a) { return a >= ZK_P ? a - ZK_P : a; }
__host__ __device__ constexpr uint64_t cx_add_mod(uint64_t a, uint64_t b) {  // a, b < p
    return a >= ZK_P - b ? a - (ZK_P - b) : a + b;
}
__host__ __device__ constexpr uint64_t cx_sub_mod(uint64_t a, uint64_t b) { return a >= b ? a - b : a + (ZK_P - b); }
constexpr uint64_t cx_mul_mod(uint64_t a, uint64_t b) {  // a < p, any b
    uint64_t r = 0;
    for (int i = 63; i >= 0; i--) {
        r = cx_add_mod(r, r);
        if (b >> i & 1) r = cx_add_mod(r, a);
    }
    return r;
}
constexpr uint64_t cx_mont(uint64_t a) { return cx_mul_mod(0xffffffffull, cx_canon(a)); }  // a 2^64 mod p

struct RcTable {
    uint64_t v[360];
};

// Circulant layers C[r][k] = c[(k - r) mod 12] plus diag(d, 0, ..., 0).  In 6x6
// blocks C = [[A, B], [B, A]], so with u = x_lo + x_hi and w = x_lo - x_hi
// (x_lo = lanes 0-5, x_hi = lanes 6-11),
//   2 (C x)_lo = (A + B) u + (A - B) w,   2 (C x)_hi = (A + B) u - (A - B) w,
// which takes 72 multiply-adds per half-vector instead of 144.  The products of
// such matrices split the same way, with (A + B)^2 and (A - B)^2.  u and w are
// formed by integer adds that leave a ready word pair; w carries an offset of
// 2^32 to stay non-negative, which the constants added to the results take
// out again (circ_offset).
template <class H>
struct Circ {  // H::c(j), j in 0..11: the first row; H::d0(): the diagonal term
    __host__ __device__ static constexpr int at(int j) { return H::c(((j % 12) + 12) % 12); }
    struct Row {
        int v[12];
    };
    static constexpr Row power_row(int n) {  // first row of C^n
        Row p{};
        for (int j = 0; j < 12; j++) p.v[j] = H::c(j);
        for (; n > 1; n--) {
            Row t{};
            for (int i = 0; i < 12; i++)
                for (int j = 0; j < 12; j++) t.v[(i + j) % 12] += p.v[i] * H::c(j);
            p = t;
        }
        return p;
    }
    template <int N>
    __host__ __device__ static constexpr int atn(int j) {
        constexpr Row p = power_row(N);
        return p.v[((j % 12) + 12) % 12];
    }
    // entries of A + B (less kappa, a multiple of the all-ones matrix) and A - B, of C^N
    template <int N>
    __host__ __device__ static constexpr int p(int r, int k) {
        return atn<N>(k - r) + atn<N>(k + 6 - r) - kappa<N>();
    }
    template <int N>
    __host__ __device__ static constexpr int q(int r, int k) {
        return atn<N>(k - r) - atn<N>(k + 6 - r);
    }
    // 2^18 times 2^33 is what fits: the entries of C^3 only do once most of their
    // common value is taken out (any even number will do; near the median, least is left)
    template <int N>
    __host__ __device__ static constexpr int kappa() {
        if constexpr (N == 3) return H::kappa3();
        else return 0;
    }
    // A + B is a 6x6 circulant [[E, F], [F, E]]: the same split once more, with
    // E + F on u_i + u_(i+3) and E - F on u_i - u_(i+3)
    template <int N>
    __host__ __device__ static constexpr double ps(int r, int k) {
        return p<N>(r, k) + p<N>(r, k + 3);
    }
    template <int N>
    __host__ __device__ static constexpr double pd(int r, int k) {
        return p<N>(r, k) - p<N>(r, k + 3);
    }
    // what the offset of w adds to output row r of either half-vector
    template <int N>
    static constexpr int64_t offset(int r) {
        int64_t v = 0;
        for (int k = 0; k < 6; k++) v += q<N>(r % 6, k);
        return (r < 6 ? v : -v) * (1ll << 31);
    }
};

// The starting values (lo, hi) of an output's two accumulators, as integers:
// lo + hi 2^32 = k (mod p), less the w offset; `bias` keeps both accumulators
// positive throughout.
struct KPair {
    uint64_t lo, hi;
};
constexpr KPair make_kpair(uint64_t k, int64_t offset, uint64_t bias) {
    const uint64_t b2 = cx_add_mod(cx_canon(bias), cx_mul_mod(cx_canon(bias), 1ull << 32));
    const uint64_t d = cx_sub_mod(cx_canon(k), b2);
    return KPair{bias - (uint64_t)offset + (d & 0xffffffffull), bias - (uint64_t)offset + (d >> 32)};
}

__device__ __forceinline__ double int_dbl(uint64_t n) { return __longlong_as_double((long long)n); }
__device__ __forceinline__ double word_dbl(uint32_t x) { return __hiloint2double(0, (int)x); }
__device__ __forceinline__ uint64_t dbl_int(double v) { return (uint64_t)__double_as_longlong(v); }
// a + b and a - b + 2^32 as doubles
__device__ __forceinline__ double sum_dbl(uint32_t a, uint32_t b) {
    uint32_t lo, hi;
    asm("add.cc.u32 %0, %2, %3;\n\taddc.u32 %1, 0, 0;" : "=r"(lo), "=r"(hi) : "r"(a), "r"(b));
    return __hiloint2double((int)hi, (int)lo);
}
__device__ __forceinline__ double diff_dbl(uint32_t a, uint32_t b) {
    uint32_t lo, hi;
    asm("sub.cc.u32 %0, %2, %3;\n\tsubc.u32 %1, 1, 0;" : "=r"(lo), "=r"(hi) : "r"(a), "r"(b));
    return __hiloint2double((int)hi, (int)lo);
}
__device__ __forceinline__ uint32_t half_of(uint64_t x, int h) { return h ? (uint32_t)(x >> 32) : (uint32_t)x; }

// Half h of the lanes as the split takes it: w, and u or (H::split3) its sums
// and differences u_i + u_(i+3), u_i - u_(i+3).
struct CircIn {
    double u[6], w[6];
};
template <class H>
__device__ __forceinline__ CircIn circ_in(const uint64_t s[12], int h) {
    CircIn x;
#pragma unroll
    for (int i = 2; i >= 0; i--) {
        const double a = sum_dbl(half_of(s[i], h), half_of(s[i + 6], h));
        const double b = sum_dbl(half_of(s[i + 3], h), half_of(s[i + 9], h));
        x.u[i] = H::split3() ? a + b : a;
        x.u[i + 3] = H::split3() ? a - b : b;
        x.w[i] = diff_dbl(half_of(s[i], h), half_of(s[i + 6], h));
        x.w[i + 3] = diff_dbl(half_of(s[i + 3], h), half_of(s[i + 9], h));
    }
    return x;
}
// f(r, value) for the 12 rows of C^N x + k (+ t / 4 on every row); lane 0, the
// last to leave an S-box, comes last in every sum.
template <class H, int N, class F>
__device__ __forceinline__ void circ_rows(const CircIn &x, const uint64_t *k, double t, F &&f) {
    using C = Circ<H>;
    if constexpr (!H::split3()) {
#pragma unroll
        for (int r = 0; r < 6; r++) {
            double pa = (double)C::template p<N>(r, 0) * x.u[0], qa = (double)C::template q<N>(r, 0) * x.w[0];
#pragma unroll
            for (int c = 1; c < 6; c++) {
                pa = fma((double)C::template p<N>(r, c), x.u[c], pa);
                qa = fma((double)C::template q<N>(r, c), x.w[c], qa);
            }
            f(r, fma(0.5, pa + qa, int_dbl(k[r])));
            f(r + 6, fma(0.5, pa - qa, int_dbl(k[r + 6])));
        }
        return;
    }
#pragma unroll
    for (int r = 0; r < 3; r++) {
        double sp = N == 3 ? fma(C::template ps<N>(r, 2), x.u[2], t) : C::template ps<N>(r, 2) * x.u[2];
        double sm = C::template pd<N>(r, 2) * x.u[5];
#pragma unroll
        for (int c = 1; c >= 0; c--) {
            sp = fma(C::template ps<N>(r, c), x.u[c], sp);
            sm = fma(C::template pd<N>(r, c), x.u[c + 3], sm);
        }
#pragma unroll
        for (int e = 0; e < 2; e++) {  // rows r and r + 3 of A + B: 2 (A + B) u = sp +- sm
            const int rr = r + 3 * e;
            const double pa = e ? sp - sm : sp + sm;
            double qa = (double)(2 * C::template q<N>(rr, 5)) * x.w[5];
#pragma unroll
            for (int c = 4; c >= 0; c--) qa = fma((double)(2 * C::template q<N>(rr, c)), x.w[c], qa);
            f(rr, fma(0.25, pa + qa, int_dbl(k[rr])));
            f(rr + 6, fma(0.25, pa - qa, int_dbl(k[rr + 6])));
        }
    }
}
// 4 times row 0 of C^N x
template <class H, int N>
__device__ __forceinline__ double circ_row0(const CircIn &x) {
    using C = Circ<H>;
    double a = C::template ps<N>(0, 2) * x.u[2], b = C::template pd<N>(0, 2) * x.u[5];
    double c = (double)(2 * C::template q<N>(0, 5)) * x.w[5];
#pragma unroll
    for (int i = 4; i > 0; i--) c = fma((double)(2 * C::template q<N>(0, i)), x.w[i], c);
    a = fma(C::template ps<N>(0, 1), x.u[1], a);
    b = fma(C::template pd<N>(0, 1), x.u[4], b);
    a = fma(C::template ps<N>(0, 0), x.u[0], a);
    b = fma(C::template pd<N>(0, 0), x.u[3], b);
    c = fma((double)(2 * C::template q<N>(0, 0)), x.w[0], c);
    return (a + b) + c;
}

template <class H>
__device__ __forceinline__ void circ_layer(uint64_t s[12], const uint64_t (*k)[12]) {
    double lo[12];
    {
        const CircIn x = circ_in<H>(s, 0);
        circ_rows<H, 1>(x, k[0], 0.0, [&](int r, double v) { lo[r] = v; });
        if (H::d0() != 0) lo[0] = fma((double)H::d0(), word_dbl((uint32_t)s[0]), lo[0]);
    }
    const uint64_t x0 = s[0];
    const CircIn x = circ_in<H>(s, 1);
    circ_rows<H, 1>(x, k[1], 0.0, [&](int r, double v) {
        if (H::d0() != 0 && r == 0) v = fma((double)H::d0(), word_dbl((uint32_t)(x0 >> 32)), v);
        s[r] = pr_reduce_split(dbl_int(lo[r]), dbl_int(v));
    });
}

// ------------------------------------------------------------ Poseidon
// MDS = C + diag(8, 0, ..., 0), C circulant.
struct PoseidonMds {
    __host__ __device__ static constexpr int c(int j) {
        constexpr uint32_t circ[12] = {ZK_POSEIDON_MDS_CIRC_LIST};
        return (int)circ[j];
    }
    __host__ __device__ static constexpr int d0() {
        constexpr uint32_t diag[12] = {ZK_POSEIDON_MDS_DIAG_LIST};
        return (int)diag[0];
    }
    __host__ __device__ static constexpr int kappa3() { return 2755704; }
    __host__ __device__ static constexpr bool split3() { return true; }
};
using PoseidonCirc = Circ<PoseidonMds>;
constexpr bool diag_only_lane0() {
    constexpr uint32_t diag[12] = {ZK_POSEIDON_MDS_DIAG_LIST};
    for (int i = 1; i < 12; i++)
        if (diag[i]) return false;
    return true;
}
static_assert(diag_only_lane0(), "the MDS layer below assumes diag(d, 0, ..., 0)");

// Round r adds its 12 constants, applies x^7 (all lanes in rounds 0-3 and
// 26-29, lane 0 otherwise) and the MDS layer M = C + d e0 e0^T.  Constants of
// round r + 1 are added inside round r's layer.
//
// The 22 partial rounds run several at a time, so that one layer's work covers
// them.  Two rounds, with x the state, x0' = S(x0), c, c' the next rounds'
// constants, y0 = (M x')_0 + c_0 and y0' = S(y0):
//   M (M x' + c + (y0' - y0) e0) + c'
//     = C^2 x' + g C e0 + d y0' e0 + (C c + c'),    g = d x0' + y0' - y0,
// plus one row for y0 and one column for g.  Three rounds go on from there with
// z0 = (C^2 x')_0 + g C_00 + d y0' + .., z0' = S(z0) and g' = d y0' + z0' - z0:
//     = C^3 x' + g C^2 e0 + g' C e0 + d z0' e0 + (C^2 c + C c' + c'').
// C^2 has row sums of 2^16; those of C^3 are 2^24, and with halves of 2^33 only
// its entries less their common part kappa / 2 stay exact (sums below 2^53):
// kappa / 2 times the sum of the lanes is formed mod p and added to every row.
// One thread per hash, bound by issue slots, takes three rounds at a time
// (rounds 4-24, and 25 alone); the forms on several threads, bound by latency,
// take two, whose dependent chain is the same length per round.
struct PoseidonTab {          // one thread per hash
    uint64_t full[9][2][12];  // layers of rounds 0-3 and 25-29 (no constants after 29)
    uint64_t trip[7][2][12];  // layers of rounds (4, 5, 6) .. (22, 23, 24)
    uint64_t mid[7][2][2];    // y0 and z0 of each
    uint64_t rc0[12];         // round 0, added before the first S-box
};
struct PoseidonGroupTab {      // several threads per hash
    uint64_t full[8][2][12];   // layers of rounds 0-3 and 26-29
    uint64_t pair[11][2][12];  // layers of round pairs (4, 5) .. (24, 25)
    uint64_t mid[11][2];       // y0 of each pair
    uint64_t rc0[12];
    // the six-thread form's rows t of A + B and A - B (for C and C^2), and C e0 at rows t and t + 6
    double rows[6][26];
};
constexpr uint64_t kFullBias = 1ull << 40;  // above the w offset of C: 34 * 2^31
constexpr uint64_t kPairBias = 1ull << 48;  // above 41 * 2^42 of -g and the w offset of C^2
constexpr uint64_t kTripBias = 1ull << 49;  // above 2^33 times the negative entries of (C^3 - kappa / 2)
struct Vec12 {
    uint64_t v[12];
};
constexpr Vec12 circ_times(const Vec12 &x) {  // C x mod p
    Vec12 y{};
    for (int r = 0; r < 12; r++)
        for (int j = 0; j < 12; j++)
            y.v[r] = cx_add_mod(y.v[r], cx_mul_mod(x.v[j], (uint64_t)PoseidonCirc::at(j - r)));
    return y;
}
constexpr Vec12 plus_rc(const Vec12 &x, const RcTable &rc, int rnd) {  // x + round rnd's constants
    Vec12 y{};
    for (int i = 0; i < 12; i++) y.v[i] = cx_add_mod(x.v[i], rnd < 30 ? cx_canon(rc.v[12 * rnd + i]) : 0);
    return y;
}
template <int N>
constexpr void put_layer(uint64_t (&to)[2][12], const Vec12 &k, uint64_t bias) {
    for (int r = 0; r < 12; r++) {
        const KPair p = make_kpair(k.v[r], PoseidonCirc::offset<N>(r), bias);
        to[0][r] = p.lo;
        to[1][r] = p.hi;
    }
}
constexpr PoseidonTab make_poseidon_tab(RcTable rc) {
    PoseidonTab t{};
    for (int i = 0; i < 12; i++) t.rc0[i] = cx_canon(rc.v[i]);
    for (int f = 0; f < 9; f++) put_layer<1>(t.full[f], plus_rc(Vec12{}, rc, (f < 4 ? f : 21 + f) + 1), kFullBias);
    for (int q = 0; q < 7; q++) {
        const int rnd = 4 + 3 * q;
        const Vec12 c = plus_rc(Vec12{}, rc, rnd + 1), c2 = plus_rc(circ_times(c), rc, rnd + 2),
                    c3 = plus_rc(circ_times(c2), rc, rnd + 3);
        const KPair y = make_kpair(c.v[0], PoseidonCirc::offset<1>(0), kFullBias);
        const KPair z = make_kpair(c2.v[0], PoseidonCirc::offset<2>(0), kFullBias << 5);
        t.mid[q][0][0] = y.lo;
        t.mid[q][0][1] = y.hi;
        t.mid[q][1][0] = z.lo;
        t.mid[q][1][1] = z.hi;
        put_layer<3>(t.trip[q], c3, kTripBias);
    }
    return t;
}
constexpr PoseidonGroupTab make_poseidon_group_tab(RcTable rc) {
    PoseidonGroupTab t{};
    for (int i = 0; i < 12; i++) t.rc0[i] = cx_canon(rc.v[i]);
    for (int f = 0; f < 8; f++) put_layer<1>(t.full[f], plus_rc(Vec12{}, rc, (f < 4 ? f : 22 + f) + 1), kFullBias);
    for (int q = 0; q < 11; q++) {
        const int rnd = 4 + 2 * q;
        const Vec12 c = plus_rc(Vec12{}, rc, rnd + 1);
        const KPair y = make_kpair(c.v[0], PoseidonCirc::offset<1>(0), kFullBias);
        t.mid[q][0] = y.lo;
        t.mid[q][1] = y.hi;
        put_layer<2>(t.pair[q], plus_rc(circ_times(c), rc, rnd + 2), kPairBias);
    }
    for (int r = 0; r < 6; r++) {
        for (int k = 0; k < 6; k++) {
            t.rows[r][k] = PoseidonCirc::p<1>(r, k);
            t.rows[r][6 + k] = PoseidonCirc::q<1>(r, k);
            t.rows[r][12 + k] = PoseidonCirc::p<2>(r, k);
            t.rows[r][18 + k] = PoseidonCirc::q<2>(r, k);
        }
        t.rows[r][24] = PoseidonCirc::at(-r);
        t.rows[r][25] = PoseidonCirc::at(-r - 6);
    }
    return t;
}

// The round tables of one hasher.  Permutations read them from the
// __constant__ bank (kernels with many resident warps keep it hot) or from a
// block's shared-memory copy of the __device__ twin (latency-bound kernels
// with a few warps, which would otherwise wait on a constant-cache miss in
// every round).
struct Poseidon2Tab {
    uint64_t rc[31][12];  // constants added after each layer: [r] before round r's S-box, [30] zero
    uint64_t diag[12];    // internal-layer diagonal, times 2^64
};
struct KeccakTab {};
constexpr Poseidon2Tab make_poseidon2_tab(RcTable rc) {
    Poseidon2Tab t{};
    for (int i = 0; i < 360; i++) t.rc[i / 12][i % 12] = cx_canon(rc.v[i]);
    constexpr uint64_t d[12] = {ZK_POSEIDON2_DIAG_LIST};
    for (int i = 0; i < 12; i++) t.diag[i] = cx_mont(d[i]);
    return t;
}
__constant__ PoseidonTab c_poseidon = make_poseidon_tab(RcTable{{ZK_POSEIDON_RC_LIST}});
__constant__ Poseidon2Tab c_poseidon2 = make_poseidon2_tab(RcTable{{ZK_POSEIDON2_RC_LIST}});
__device__ PoseidonGroupTab g_poseidon = make_poseidon_group_tab(RcTable{{ZK_POSEIDON_RC_LIST}});
__device__ Poseidon2Tab g_poseidon2 = make_poseidon2_tab(RcTable{{ZK_POSEIDON2_RC_LIST}});
__constant__ uint64_t c_keccak_rc[24] = {ZK_KECCAK_RC_LIST};
__constant__ KeccakTab c_keccak_tab;

// Three partial rounds (the triple q), see above.
__device__ __forceinline__ void poseidon_triple(uint64_t s[12], int q, const PoseidonTab &tab) {
    using C = PoseidonCirc;
    constexpr double d0 = (double)PoseidonMds::d0(), c00 = (double)C::at(0);
    s[0] = pr_pow7(s[0]);
    const uint64_t x0 = s[0];
    CircIn x[2];
    double y[2], z[2], tau[2], g0[2], g1[2], zp[2], lo[12];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        x[h] = circ_in<PoseidonMds>(s, h);
        y[h] = fma(0.25, circ_row0<PoseidonMds, 1>(x[h]), fma(d0, word_dbl(half_of(x0, h)), int_dbl(tab.mid[q][0][h])));
        z[h] = fma(0.25, circ_row0<PoseidonMds, 2>(x[h]), int_dbl(tab.mid[q][1][h]));
        tau[h] = x[h].u[2] + x[h].u[1] + x[h].u[0];
    }
    const uint64_t yr = pr_reduce_split(dbl_int(y[0]), dbl_int(y[1])), yp = pr_pow7(yr);
    // kappa / 2 times the sum of the lanes, mod p
    const uint64_t sum = pr_reduce_split(dbl_int(tau[0]), dbl_int(tau[1]));
    constexpr double k2 = (double)(C::kappa<3>() / 2);
    const uint64_t t = pr_reduce_split(dbl_int(k2 * word_dbl((uint32_t)sum)), dbl_int(k2 * word_dbl((uint32_t)(sum >> 32))));
#pragma unroll
    for (int h = 0; h < 2; h++) {
        g0[h] = fma(d0, word_dbl(half_of(x0, h)), word_dbl(half_of(yp, h)) - word_dbl(half_of(yr, h)));
        z[h] = fma(c00, g0[h], fma(d0, word_dbl(half_of(yp, h)), z[h]));
    }
    const uint64_t zr = pr_reduce_split(dbl_int(z[0]), dbl_int(z[1])), zq = pr_pow7(zr);
#pragma unroll
    for (int h = 0; h < 2; h++) {
        zp[h] = word_dbl(half_of(zq, h));
        g1[h] = fma(d0, word_dbl(half_of(yp, h)), zp[h] - word_dbl(half_of(zr, h)));
        circ_rows<PoseidonMds, 3>(x[h], tab.trip[q][h], 4.0 * word_dbl(half_of(t, h)), [&](int r, double v) {
            v = fma((double)C::atn<2>(-r), g0[h], v);
            v = fma((double)C::at(-r), g1[h], v);
            if (r == 0) v = fma(d0, zp[h], v);
            if (h == 0) lo[r] = v;
            else s[r] = pr_reduce_split(dbl_int(lo[r]), dbl_int(v));
        });
    }
}

// x^7 on all 12 lanes.  W = 4: three passes over 4 lanes with a rotation
// between them (a small loop body, and so a small instruction footprint, for
// kernels with many resident warps).  W = 12: all lanes at once (more
// independent work in flight, for kernels whose few warps wait on latency).
template <int W = 4>
__device__ __forceinline__ void pow7_all(uint64_t s[12]) {
    if constexpr (W == 12) {
#pragma unroll
        for (int i = 0; i < 12; i++) s[i] = pr_pow7(s[i]);
    } else {
#pragma unroll 1
        for (int q = 0; q < 3; q++) {
#pragma unroll
            for (int i = 0; i < 4; i++) s[i] = pr_pow7(s[i]);
            const uint64_t t0 = s[0], t1 = s[1], t2 = s[2], t3 = s[3];
#pragma unroll
            for (int i = 0; i < 8; i++) s[i] = s[i + 4];
            s[8] = t0;
            s[9] = t1;
            s[10] = t2;
            s[11] = t3;
        }
    }
}

// The permutation on a partially reduced state (outputs partially reduced).
template <int W = 4>
__device__ __forceinline__ void poseidon_permute(uint64_t s[12], const PoseidonTab &tab = c_poseidon) {
#pragma unroll
    for (int i = 0; i < 12; i++) s[i] = pr_add_c(s[i], tab.rc0[i]);
#pragma unroll 1
    for (int half = 0; half < 2; half++) {
#pragma unroll 1
        for (int f = 0; f < 4 + half; f++) {
            if (half && f == 0) s[0] = pr_pow7(s[0]);  // round 25
            else pow7_all<W>(s);
            circ_layer<PoseidonMds>(s, tab.full[4 * half + f]);
        }
        if (half) break;
#pragma unroll 1
        for (int q = 0; q < 7; q++) poseidon_triple(s, q, tab);
    }
}

// ----------------------------------------------------------- Poseidon2
// External layer = (I + [1 1 1] (x) I_4) * blockdiag(M4, M4, M4) with
// M4 = [[5,7,1,3],[4,6,1,1],[1,3,5,7],[1,1,4,6]] (poseidon2.cu:64-110):
// y_b = M4 x_b per 4-lane block, then out_b = y_b + (y_0 + y_1 + y_2).
// M4 x is the 8-addition network of the Poseidon2 paper (Grassi, Khovratovich,
// Schofnegger 2023, section 5.1): t0 = x0 + x1, t1 = x2 + x3, t2 = 2 x1 + t1,
// t3 = 2 x3 + t0, t4 = 4 t1 + t3, t5 = 4 t0 + t2, M4 x = (t3 + t5, t5, t2 + t4, t4).
__device__ __forceinline__ void poseidon2_external_half(const uint64_t s[12], int h, double o[12]) {
    double y[12];
#pragma unroll
    for (int b = 0; b < 3; b++) {
        const uint32_t x0 = half_of(s[4 * b], h), x1 = half_of(s[4 * b + 1], h);
        const uint32_t x2 = half_of(s[4 * b + 2], h), x3 = half_of(s[4 * b + 3], h);
        const double t0 = sum_dbl(x0, x1), t1 = sum_dbl(x2, x3);
        const double t2 = fma(2.0, word_dbl(x1), t1), t3 = fma(2.0, word_dbl(x3), t0);
        const double t4 = fma(4.0, t1, t3), t5 = fma(4.0, t0, t2);
        y[4 * b] = t3 + t5;
        y[4 * b + 1] = t5;
        y[4 * b + 2] = t2 + t4;
        y[4 * b + 3] = t4;
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const double sm = (y[j] + y[4 + j]) + y[8 + j];
#pragma unroll
        for (int b = 0; b < 3; b++) o[4 * b + j] = y[4 * b + j] + sm;
    }
}
__device__ __forceinline__ void poseidon2_external(uint64_t s[12], const uint64_t *c) {
    double lo[12], hi[12];
    poseidon2_external_half(s, 0, lo);
    poseidon2_external_half(s, 1, hi);
#pragma unroll
    for (int r = 0; r < 12; r++) s[r] = pr_reduce_split_add(dbl_int(lo[r]), dbl_int(hi[r]), c[r]);
}

// Internal layer, x_i <- x_i D_i + sum_j x_j (poseidon2.cu:131-146), and the
// next round's constant (lane 0 only).  With R = 2^64, each lane is one
// Montgomery reduction of x_i (D_i R) + (sum R mod p): the sum's two words
// start the product's accumulators (mul_add_words), so adding it costs nothing
// per lane.  R = 2^32 - 1 and 2^128 = -2^32, so (z2 z1 z0) R = (z0 - z2) 2^32 - z0 - z1.
__device__ __forceinline__ uint64_t poseidon2_sum_mont(uint32_t z0, uint32_t z1, uint32_t z2) {
    // z0 2^32 + (2^64 - 2^32 + 1) [= p] - z0 - z1 - z2 2^32, positive and below 2^65
    uint32_t r0, r1;
    asm("{\n\t"
        ".reg .u32 a0, a1, b0, b1, k;\n\t"
        "add.cc.u32 b0, %2, %3;\n\t"       // z0 + z1 + z2 2^32
        "addc.u32 b1, %4, 0;\n\t"
        "sub.cc.u32 a0, 0, b0;\n\t"        // z0 2^32 - that; a borrow adds p back
        "subc.cc.u32 a1, %2, b1;\n\t"
        "subc.u32 k, 0, 0;\n\t"
        "sub.cc.u32 %0, a0, k;\n\t"
        "subc.u32 %1, a1, 0;\n\t"
        "}"
        : "=r"(r0), "=r"(r1)
        : "r"(z0), "r"(z1), "r"(z2));
    return ((uint64_t)r1 << 32) | r0;
}
__device__ __forceinline__ uint64_t poseidon2_lane(uint64_t x, uint64_t d, uint64_t sum) {
    uint32_t w[4];
    mul_add_words(x, d, (uint32_t)sum, (uint32_t)(sum >> 32), w);
    return mont_reduce(w[0], w[1], w[2], w[3]);
}
__device__ __forceinline__ void poseidon2_internal(uint64_t s[12], uint64_t c0, const uint64_t *diag) {
    uint32_t z0 = (uint32_t)s[0], z1 = (uint32_t)(s[0] >> 32), z2 = 0;  // the sum of the lanes, exact in 96 bits
#pragma unroll
    for (int i = 1; i < 12; i++) {
        asm("add.cc.u32 %0, %0, %3;\n\t"
            "addc.cc.u32 %1, %1, %4;\n\t"
            "addc.u32 %2, %2, 0;"
            : "+r"(z0), "+r"(z1), "+r"(z2)
            : "r"((uint32_t)s[i]), "r"((uint32_t)(s[i] >> 32)));
    }
    const uint64_t sum = poseidon2_sum_mont(z0, z1, z2);
#pragma unroll
    for (int i = 0; i < 12; i++) s[i] = poseidon2_lane(s[i], diag[i], sum);
    s[0] = pr_add_c(s[0], c0);
}

template <int W = 4>
__device__ __forceinline__ void poseidon2_permute(uint64_t s[12], const Poseidon2Tab &tab = c_poseidon2) {
    poseidon2_external(s, tab.rc[0]);
#pragma unroll 1
    for (int half = 0; half < 2; half++) {
#pragma unroll 1
        for (int f = 0; f < 4; f++) {
            pow7_all<W>(s);
            // after rounds 0-2 and 26-28 the next round's constants, after round 3 those of the
            // first internal round (lane 0), none after the last
            poseidon2_external(s, tab.rc[26 * half + f + 1]);
        }
        if (half) break;
        // internal rounds: only lane 0 of their constants is non-zero
#pragma unroll 1
        for (int rnd = 4; rnd < 26; rnd++) {
            s[0] = pr_pow7(s[0]);
            poseidon2_internal(s, tab.rc[rnd + 1][0], tab.diag);
        }
#pragma unroll
        for (int i = 1; i < 12; i++) s[i] = pr_add_c(s[i], tab.rc[26][i]);
    }
}

// --------------------------------------------------------------- Keccak
// Keccak-f on 32-bit halves with each three-input operation written as one
// lop3 and each rotation as two funnel shifts: 180 operations a round (theta
// 80, rho 48, chi 50, iota 2), all on the ALU pipe, which bounds it (97 % busy
// already from 64-bit words).  Tree 2^18 x 135: 0.771 -> 0.645 ms.
__device__ __forceinline__ uint32_t xor3(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0x96;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
    return r;
}
__device__ __forceinline__ uint32_t chi3(uint32_t a, uint32_t b, uint32_t c) {  // a ^ (~b & c)
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xd2;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
    return r;
}
template <int S>
__device__ __forceinline__ void rotl_words(uint32_t &o0, uint32_t &o1, uint32_t l, uint32_t h) {
    if constexpr (S == 0) o0 = l, o1 = h;
    else if constexpr (S < 32) o0 = __funnelshift_l(h, l, S), o1 = __funnelshift_l(l, h, S);
    else o0 = __funnelshift_l(l, h, S - 32), o1 = __funnelshift_l(h, l, S - 32);
}
template <int I>
__device__ __forceinline__ void keccak_rho_pi(const uint32_t l[25], const uint32_t h[25], uint32_t bl[25], uint32_t bh[25]) {
    if constexpr (I < 25) {
        constexpr int rho[25] = {ZK_KECCAK_RHO_LIST};
        constexpr int x = I % 5, y = I / 5, d = y + 5 * ((2 * x + 3 * y) % 5);
        rotl_words<rho[I]>(bl[d], bh[d], l[I], h[I]);
        keccak_rho_pi<I + 1>(l, h, bl, bh);
    }
}
__device__ __forceinline__ void keccak_f1600(uint64_t a[25]) {
    uint32_t l[25], h[25];
#pragma unroll
    for (int i = 0; i < 25; i++) l[i] = (uint32_t)a[i], h[i] = (uint32_t)(a[i] >> 32);
#pragma unroll 1
    for (int rnd = 0; rnd < 24; rnd++) {
        uint32_t cl[5], ch[5], bl[25], bh[25];
#pragma unroll
        for (int x = 0; x < 5; x++) {
            cl[x] = xor3(xor3(l[x], l[x + 5], l[x + 10]), l[x + 15], l[x + 20]);
            ch[x] = xor3(xor3(h[x], h[x + 5], h[x + 10]), h[x + 15], h[x + 20]);
        }
#pragma unroll
        for (int x = 0; x < 5; x++) {
            uint32_t fl, fh;
            rotl_words<1>(fl, fh, cl[(x + 1) % 5], ch[(x + 1) % 5]);
#pragma unroll
            for (int y = 0; y < 25; y += 5) {
                l[x + y] = xor3(l[x + y], cl[(x + 4) % 5], fl);
                h[x + y] = xor3(h[x + y], ch[(x + 4) % 5], fh);
            }
        }
        // rho + pi: B[y, 2x + 3y] = rot(A[x, y], rho[x, y])
        keccak_rho_pi<0>(l, h, bl, bh);
        // chi
#pragma unroll
        for (int y = 0; y < 25; y += 5)
#pragma unroll
            for (int x = 0; x < 5; x++) {
                l[x + y] = chi3(bl[x + y], bl[(x + 1) % 5 + y], bl[(x + 2) % 5 + y]);
                h[x + y] = chi3(bh[x + y], bh[(x + 1) % 5 + y], bh[(x + 2) % 5 + y]);
            }
        l[0] ^= (uint32_t)c_keccak_rc[rnd];
        h[0] ^= (uint32_t)(c_keccak_rc[rnd] >> 32);
    }
#pragma unroll
    for (int i = 0; i < 25; i++) a[i] = ((uint64_t)h[i] << 32) | l[i];
}

// --------------------------------------------------------------- Monolith
// Monolith-64, width 12, 6 rounds (native/monolith/monolith.cu:117-233):
// concrete(rc_0), then per round r = 1..6: bars, bricks, concrete(rc_r).
//  * concrete: the circulant matrix (row r column c = ROW[(c - r) mod 12], row
//    sum 160) plus the round constant, mod p.  The same exact FP64 split as
//    the Poseidon MDS, no diagonal.  Lanes 0-3 are canonicalised afterwards:
//    the Bar S-box acts on the bits of the canonical value.
//  * bars: Bar on every byte of lanes 0-3,
//    y = rotl1(x ^ (rotl1(~x) & rotl2(x) & rotl3(x))) (rotations within the byte).
//  * bricks (Feistel type 3): lane i, from 11 down to 1, += (lane i-1)^2 mod p,
//    the square of lane i-1 before the layer.  zeknox keeps that sum as a
//    65-bit value for the next concrete layer; here it is taken mod p
//    (pr_sqr_add), which is the same field element.
struct MonolithMds {
    __host__ __device__ static constexpr int c(int j) {
        constexpr uint32_t row[12] = {ZK_MONOLITH_MDS_ROW_LIST};
        return (int)row[j];
    }
    __host__ __device__ static constexpr int d0() { return 0; }
    // its bytewise Bars keep the integer pipes busiest: the further split measured 1 % slower
    __host__ __device__ static constexpr bool split3() { return false; }
};

// Accumulator starting values of the 7 concrete layers.
struct MonolithTab {
    uint64_t k[7][2][12];
};
constexpr MonolithTab make_monolith_tab() {
    MonolithTab t{};
    constexpr uint64_t rc[84] = {ZK_MONOLITH_RC_LIST};
    for (int rnd = 0; rnd < 7; rnd++)
        for (int r = 0; r < 12; r++) {
            const KPair k = make_kpair(rc[12 * rnd + r], Circ<MonolithMds>::offset<1>(r), kFullBias);
            t.k[rnd][0][r] = k.lo;
            t.k[rnd][1][r] = k.hi;
        }
    return t;
}
__constant__ MonolithTab c_monolith = make_monolith_tab();
__device__ MonolithTab g_monolith = make_monolith_tab();

__device__ __forceinline__ void monolith_concrete(uint64_t s[12], const uint64_t (*k)[12]) {
    circ_layer<MonolithMds>(s, k);
#pragma unroll
    for (int r = 0; r < 4; r++) s[r] = gl_canon(s[r]);
}

// Rotate every byte of x left by K (within the byte).
template <int K>
__device__ __forceinline__ uint32_t rotl_bytes(uint32_t x) {
    constexpr uint32_t low = 0x01010101u * ((1u << K) - 1u);  // the low K bits of each byte
    return ((x << K) & ~low) | ((x >> (8 - K)) & low);
}
__device__ __forceinline__ uint32_t monolith_bar32(uint32_t x) {
    return rotl_bytes<1>(x ^ (rotl_bytes<1>(~x) & rotl_bytes<2>(x) & rotl_bytes<3>(x)));
}

__device__ __forceinline__ void monolith_permute(uint64_t s[12], const MonolithTab &tab = c_monolith) {
    monolith_concrete(s, tab.k[0]);
#pragma unroll 1
    for (int rnd = 1; rnd <= 6; rnd++) {
#pragma unroll
        for (int i = 0; i < 4; i++)
            s[i] = ((uint64_t)monolith_bar32((uint32_t)(s[i] >> 32)) << 32) | monolith_bar32((uint32_t)s[i]);
#pragma unroll
        for (int i = 11; i > 0; i--) s[i] = pr_sqr_add(s[i - 1], s[i]);
        monolith_concrete(s, tab.k[rnd]);
    }
}

// ---------------------------------------------------- Poseidon-BN128
// circomlib's Poseidon over the BN254 scalar field r, t = 5, 8 full and 60
// partial rounds in the optimised form (native/poseidon/poseidon_bn128.cu:
// 111-193).  The 12 Goldilocks lanes become 4 field elements x_i =
// lane[3i+2] + lane[3i+1] 2^64 + lane[3i] 2^128; the state is (0, x_0, .., x_3).
// Output lane 3i + k is limb 2 - k of state element i, reduced mod p once.
//
// A field element is nine limbs of 29 bits, in Montgomery form with R = 2^261
// (the tables hold 2^256 forms, times 2^5 here).  The 18 columns of a product
// are 64-bit sums of 58-bit products without a carry between them: 54 of them
// fit (five products of one matrix row and the nine of a reduction), so a row
// of the MDS or of a sparse matrix costs one reduction, and an addend joins in
// the upper columns.  Values are not reduced below r: a Montgomery result is
// below r plus the product over R, and the state elements that a partial round
// adds to grow by less than 1.1 r in each of the 60 rounds, to below 2^260.
// Products on carry chains of 32-bit limbs, the form before this one, left
// each warp waiting on its chain.  Trees of 135-word leaves, one thread per hash
// throughout: 8192 leaves 27.2 -> 12.5 ms, 65536 leaves 51.7 -> 33.8 ms (10.0 and
// 31.7 with the narrow levels on five threads, end of file).
constexpr int kBnL = 9;
constexpr uint32_t kBnMask = (1u << 29) - 1;
struct Fr {
    uint32_t v[kBnL];
};
struct alignas(8) BnTab {  // copied in 8-byte words
    Fr c[100];  // round constants
    Fr s[540];  // sparse partial-round matrices, 9 values per round
    Fr m[25];   // MDS, m[5 j + i] multiplies state j into lane i
    Fr p[25];   // pre-sparse matrix (same indexing)
    Fr r2;      // R^2 mod r
};
__host__ __device__ constexpr uint64_t bn_r64(int i) {  // the modulus r, little-endian words
    constexpr uint64_t r[4] = {0x43e1f593f0000001ull, 0x2833e84879b97091ull, 0xb85045b68181585dull,
                               0x30644e72e131a029ull};
    return r[i];
}
// limb i (29 bits) of a 256-bit value
__host__ __device__ constexpr uint32_t bn_limb(uint64_t w0, uint64_t w1, uint64_t w2, uint64_t w3, int i) {
    const uint64_t w[5] = {w0, w1, w2, w3, 0};
    const int b = 29 * i, q = b / 64, o = b % 64;
    return (uint32_t)((w[q] >> o) | (o > 35 ? w[q + 1] << (64 - o) : 0)) & kBnMask;
}
__host__ __device__ constexpr uint32_t bn_r(int i) { return bn_limb(bn_r64(0), bn_r64(1), bn_r64(2), bn_r64(3), i); }
constexpr uint32_t bn_ninv() {  // -r^-1 mod 2^29
    uint32_t x = 1;
    for (int i = 0; i < 6; i++) x *= 2u - bn_r(0) * x;
    return (0u - x) & kBnMask;
}
constexpr uint32_t kBnNinv = bn_ninv();
static_assert(((bn_r(0) * kBnNinv + 1) & kBnMask) == 0, "-r^-1 mod 2^29");
// 2^k x mod r as limbs, x < r in four 64-bit words
constexpr Fr bn_scaled(const uint64_t *x, int k) {
    uint64_t t[4] = {x[0], x[1], x[2], x[3]};
    for (int n = 0; n < k; n++) {
        uint64_t top = 0;
        for (int i = 0; i < 4; i++) {
            const uint64_t v = (t[i] << 1) | top;
            top = t[i] >> 63;
            t[i] = v;
        }
        bool ge = true;  // r < 2^254, so the doubled value fits 256 bits
        for (int i = 3; i >= 0; i--)
            if (t[i] != bn_r64(i)) {
                ge = t[i] > bn_r64(i);
                break;
            }
        if (ge) {
            uint64_t bw = 0;
            for (int i = 0; i < 4; i++) {
                const uint64_t d = t[i] - bn_r64(i), e = d - bw;
                bw = (t[i] < bn_r64(i)) | (d < bw);
                t[i] = e;
            }
        }
    }
    Fr f{};
    for (int i = 0; i < kBnL; i++) f.v[i] = bn_limb(t[0], t[1], t[2], t[3], i);
    return f;
}
constexpr BnTab make_bn_tab() {
    BnTab t{};
    constexpr uint64_t c[400] = {ZK_BN128_C_LIST};
    constexpr uint64_t sp[2160] = {ZK_BN128_S_LIST};
    constexpr uint64_t m[100] = {ZK_BN128_M_LIST};
    constexpr uint64_t pm[100] = {ZK_BN128_P_LIST};
    for (int i = 0; i < 100; i++) t.c[i] = bn_scaled(c + 4 * i, 5);
    for (int i = 0; i < 540; i++) t.s[i] = bn_scaled(sp + 4 * i, 5);
    for (int i = 0; i < 25; i++) t.m[i] = bn_scaled(m + 4 * i, 5);
    for (int i = 0; i < 25; i++) t.p[i] = bn_scaled(pm + 4 * i, 5);
    constexpr uint64_t r2[4] = {0x1bb8e645ae216da7ull, 0x53fe3ab1e35c59e3ull, 0x8c49833d53bb8085ull,
                                0x0216d0b17f4e44a5ull};  // 2^512 mod r
    t.r2 = bn_scaled(r2, 10);
    return t;
}
__constant__ BnTab c_bn128 = make_bn_tab();
__device__ BnTab g_bn128 = make_bn_tab();
struct BnCols {
    uint64_t c[2 * kBnL];
};
__device__ __forceinline__ void bn_acc(BnCols &t, const Fr &x, const Fr &y) {  // t += x y
#pragma unroll
    for (int i = 0; i < kBnL; i++)
#pragma unroll
        for (int j = 0; j < kBnL; j++) t.c[i + j] += (uint64_t)x.v[i] * y.v[j];
}
__device__ __forceinline__ BnCols bn_addend(const Fr &a) {  // a R
    BnCols t;
#pragma unroll
    for (int i = 0; i < kBnL; i++) {
        t.c[i] = 0;
        t.c[kBnL + i] = a.v[i];
    }
    return t;
}
__device__ __forceinline__ BnCols bn_zero() {
    BnCols t;
#pragma unroll
    for (int i = 0; i < 2 * kBnL; i++) t.c[i] = 0;
    return t;
}
// t / R mod r, limbs below 2^29
__device__ __forceinline__ Fr bn_reduce(BnCols &t) {
#pragma unroll
    for (int i = 0; i < kBnL; i++) {
        const uint32_t m = ((uint32_t)t.c[i] * kBnNinv) & kBnMask;
#pragma unroll
        for (int j = 0; j < kBnL; j++) t.c[i + j] += (uint64_t)m * bn_r(j);
        t.c[i + 1] += t.c[i] >> 29;
    }
    Fr z;
#pragma unroll
    for (int i = 0; i < kBnL; i++) {
        z.v[i] = (uint32_t)t.c[kBnL + i] & kBnMask;
        if (i + 1 < kBnL) t.c[kBnL + i + 1] += t.c[kBnL + i] >> 29;
    }
    return z;
}
__device__ __forceinline__ Fr bn_sqr(const Fr &x) {
    BnCols t = bn_zero();
#pragma unroll
    for (int i = 0; i < kBnL; i++) {
        t.c[2 * i] += (uint64_t)x.v[i] * x.v[i];
        const uint32_t d = 2 * x.v[i];
#pragma unroll
        for (int j = i + 1; j < kBnL; j++) t.c[i + j] += (uint64_t)d * x.v[j];
    }
    return bn_reduce(t);
}
__device__ __forceinline__ Fr bn_sbox_add(const Fr &x, const Fr &c) {  // x^5 + c
    const Fr x4 = bn_sqr(bn_sqr(x));
    BnCols t = bn_addend(c);
    bn_acc(t, x4, x);
    return bn_reduce(t);
}
// A full round: S-box and constants (null: none), then st <- M^T st
// (new_i = sum_j m[5 j + i] st_j).  Both run one lane per iteration with the
// state rotating through registers, so the kernel holds one copy of each.
__device__ __forceinline__ void bn_full_round(Fr st[5], const Fr *c, const Fr *m) {
#pragma unroll 1
    for (int i = 0; i < 5; i++) {
        Fr k{};
        if (c) k = c[i];
        const Fr y = bn_sbox_add(st[0], k);
#pragma unroll
        for (int j = 0; j < 4; j++) st[j] = st[j + 1];
        st[4] = y;
    }
    Fr out[5];
#pragma unroll 1
    for (int i = 0; i < 5; i++) {
        BnCols t = bn_zero();
#pragma unroll
        for (int j = 0; j < 5; j++) bn_acc(t, st[j], m[5 * j + i]);
#pragma unroll
        for (int j = 0; j < 4; j++) out[j] = out[j + 1];
        out[4] = bn_reduce(t);
    }
#pragma unroll
    for (int i = 0; i < 5; i++) st[i] = out[i];
}

// Lane words in and out: x from (lane[2], lane[1], lane[0]) in Montgomery form
// plus c, and the three low 64-bit words of a state element, canonical mod p.
__device__ __forceinline__ Fr bn_from_words(const uint64_t lane[3], const Fr &c, const BnTab &tab) {
    Fr x;
#pragma unroll
    for (int l = 0; l < kBnL; l++) x.v[l] = bn_limb(lane[2], lane[1], lane[0], 0, l);
    BnCols t = bn_addend(c);
    bn_acc(t, x, tab.r2);
    return bn_reduce(t);
}
__device__ __forceinline__ void bn_words(const Fr &x, uint64_t lane[3]) {
    BnCols t = bn_zero();
#pragma unroll
    for (int l = 0; l < kBnL; l++) t.c[l] = x.v[l];
    const Fr v = bn_reduce(t);  // out of Montgomery form, in [0, r]
    bool is_r = true;
#pragma unroll
    for (int l = 0; l < kBnL; l++) is_r = is_r && v.v[l] == bn_r(l);
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const int q = 2 - k;  // 64-bit word q of the value
        uint64_t w = 0;
#pragma unroll
        for (int l = 0; l < kBnL; l++) {
            const int sh = 29 * l - 64 * q;
            if (sh > -29 && sh < 64) w |= sh >= 0 ? (uint64_t)v.v[l] << sh : (uint64_t)v.v[l] >> -sh;
        }
        lane[k] = is_r ? 0ull : gl_canon(w);
    }
}

__device__ __forceinline__ void poseidon_bn128_permute(uint64_t s[12], const BnTab &tab = c_bn128) {
    Fr st[5];
    st[0] = tab.c[0];
#pragma unroll
    for (int i = 0; i < 4; i++) st[i + 1] = bn_from_words(s + 3 * i, tab.c[i + 1], tab);
#pragma unroll 1
    for (int half = 0; half < 2; half++) {
        // full rounds 1-4 (constants from 5 on, P after the 4th) and 5-8 (from 85 on, none after the last)
#pragma unroll 1
        for (int r = 0; r < 4; r++)
            bn_full_round(st, half ? (r < 3 ? tab.c + 85 + 5 * r : nullptr) : tab.c + 5 * (r + 1),
                          !half && r == 3 ? tab.p : tab.m);
        if (half) break;
#pragma unroll 1
        for (int r = 0; r < 60; r++) {  // partial rounds with the sparse matrices
            const Fr *sp = tab.s + 9 * r;
            const Fr x0 = bn_sbox_add(st[0], tab.c[25 + r]);
            BnCols t = bn_zero();
            bn_acc(t, x0, sp[0]);
#pragma unroll
            for (int j = 1; j < 5; j++) bn_acc(t, st[j], sp[j]);
            st[0] = bn_reduce(t);
#pragma unroll 1
            for (int k = 1; k < 5; k++) {  // lane k, the lanes rotating
                BnCols u = bn_addend(st[1]);
                bn_acc(u, x0, sp[4 + k]);
                st[1] = st[2];
                st[2] = st[3];
                st[3] = st[4];
                st[4] = bn_reduce(u);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; i++) bn_words(st[i], s + 3 * i);
}

// ------------------------------------------------------------ hashers
enum : int { kPoseidon = 0, kKeccak = 1, kPoseidonBN128 = 2, kPoseidon2 = 3, kMonolith = 4 };

// Leaf elements are reduced mod p when read (a no-op for canonical inputs).
template <int H, int W = 4>
__device__ __forceinline__ void hash_one(const uint64_t *__restrict__ in, uint32_t n, uint64_t *__restrict__ out) {
    if constexpr (H == kKeccak) {
        if (n < 4) {  // copy n words, leave the rest of the digest as it was
#pragma unroll
            for (uint32_t i = 0; i < 4; i++)
                if (i < n) out[i] = in[i];
            return;
        }
        uint64_t a[25];
#pragma unroll
        for (int i = 0; i < 25; i++) a[i] = 0;
        uint32_t idx = 0;
        for (; idx + 17 <= n; idx += 17) {
#pragma unroll
            for (int i = 0; i < 17; i++) a[i] ^= in[idx + i];
            keccak_f1600(a);
        }
        const uint32_t rem = n - idx;  // 0..16 whole words, then the pad
#pragma unroll
        for (int i = 0; i < 17; i++) {
            uint64_t w = (uint32_t)i < rem ? in[idx + i] : 0ull;
            if ((uint32_t)i == rem) w ^= 0x01ull;
            if (i == 16) w ^= 0x80ull << 56;
            a[i] ^= w;
        }
        keccak_f1600(a);
        out[0] = a[0];
        out[1] = a[1];
        out[2] = a[2];
        out[3] = a[3] & 0xffull;
    } else {
        if (n <= 4) {
#pragma unroll
            for (uint32_t i = 0; i < 4; i++) out[i] = i < n ? in[i] : 0ull;
            return;
        }
        uint64_t s[12];
#pragma unroll
        for (int i = 0; i < 12; i++) s[i] = 0;
        for (uint32_t idx = 0; idx < n; idx += 8) {
            const uint32_t len = n - idx < 8 ? n - idx : 8;
            if (len == 8) {
#pragma unroll
                for (int j = 0; j < 8; j++) s[j] = gl_canon(in[idx + j]);
            } else {
#pragma unroll
                for (int j = 0; j < 8; j++)
                    if ((uint32_t)j < len) s[j] = gl_canon(in[idx + j]);
            }
            if constexpr (H == kPoseidon) poseidon_permute<W>(s);
            else if constexpr (H == kMonolith) monolith_permute(s);
            else if constexpr (H == kPoseidonBN128) poseidon_bn128_permute(s);
            else poseidon2_permute<W>(s);
        }
        out[0] = gl_canon(s[0]);
        out[1] = gl_canon(s[1]);
        out[2] = gl_canon(s[2]);
        out[3] = gl_canon(s[3]);
    }
}

template <int H>
struct TabOf;
template <>
struct TabOf<kPoseidon> {
    using type = PoseidonTab;
};
template <>
struct TabOf<kPoseidon2> {
    using type = Poseidon2Tab;
};
template <>
struct TabOf<kKeccak> {
    using type = KeccakTab;
};
template <>
struct TabOf<kMonolith> {
    using type = MonolithTab;
};
template <>
struct TabOf<kPoseidonBN128> {
    using type = BnTab;
};
template <int H>
__device__ __forceinline__ const typename TabOf<H>::type &const_tab() {
    if constexpr (H == kPoseidon) return c_poseidon;
    else if constexpr (H == kPoseidon2) return c_poseidon2;
    else if constexpr (H == kMonolith) return c_monolith;
    else if constexpr (H == kPoseidonBN128) return c_bn128;
    else return c_keccak_tab;
}

// The tables of the forms on several threads (and of one block per subtree),
// copied to shared memory from their __device__ twin.
template <int H>
using GroupTabOf = typename std::conditional<H == kPoseidon, PoseidonGroupTab, typename TabOf<H>::type>::type;
template <int H>
__device__ __forceinline__ const GroupTabOf<H> *global_tab() {
    if constexpr (H == kPoseidon) return &g_poseidon;
    else if constexpr (H == kPoseidon2) return &g_poseidon2;
    else if constexpr (H == kMonolith) return &g_monolith;
    else if constexpr (H == kPoseidonBN128) return &g_bn128;
    else return nullptr;
}

// H(l || r) of two digests; W and tab choose the S-box width and the table copy.
template <int H, int W = 4>
__device__ __forceinline__ void hash_two(const uint64_t *l, const uint64_t *r, uint64_t *out,
                                         const typename TabOf<H>::type &tab = const_tab<H>()) {
    if constexpr (H == kKeccak) {
        // keccak256(left[0..25) || right[0..25)): 50 bytes in one block
        uint64_t a[25];
#pragma unroll
        for (int i = 0; i < 25; i++) a[i] = 0;
        const uint64_t r0 = r[0], r1 = r[1], r2 = r[2], r3 = r[3];
        a[0] = l[0];
        a[1] = l[1];
        a[2] = l[2];
        a[3] = (l[3] & 0xffull) | (r0 << 8);
        a[4] = (r0 >> 56) | (r1 << 8);
        a[5] = (r1 >> 56) | (r2 << 8);
        a[6] = (r2 >> 56) | ((r3 & 0xffull) << 8) | (0x01ull << 16);
        a[16] = 0x80ull << 56;
        keccak_f1600(a);
        out[0] = a[0];
        out[1] = a[1];
        out[2] = a[2];
        out[3] = a[3] & 0xffull;
    } else {
        uint64_t s[12];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            s[i] = gl_canon(l[i]);
            s[4 + i] = gl_canon(r[i]);
            s[8 + i] = 0;
        }
        if constexpr (H == kPoseidon) poseidon_permute<W>(s, tab);
        else if constexpr (H == kMonolith) monolith_permute(s, tab);
        else if constexpr (H == kPoseidonBN128) poseidon_bn128_permute(s, tab);
        else poseidon2_permute<W>(s, tab);
        out[0] = gl_canon(s[0]);
        out[1] = gl_canon(s[1]);
        out[2] = gl_canon(s[2]);
        out[3] = gl_canon(s[3]);
    }
}

// ------------------------------------------- Poseidon on two threads
// For trees with too few leaves to fill the GPU one thread per hash, but
// enough that six threads per hash would be issue-bound: the permutation is
// split over the two threads of a lane pair (lanes 2k, 2k + 1; sixteen hashes
// per warp, no idle lanes).  Thread h owns state lanes 6h .. 6h + 5 and
// computes half h of every layer's outputs: six 32-bit shuffles bring the
// partner's input halves, and six 64-bit shuffles hand each thread the other
// half of its own lanes' outputs.  In a pair of partial rounds lane 0's first
// S-box runs on thread 0 and its second one, after an exchange of the halves
// of y0, on both threads.  The squares are plain products here (8192 x 135 tree
// 310 -> 305 us; the six-thread form loses by that, 2048 x 135: 185 -> 230).
__device__ __forceinline__ uint32_t shfl_xor32(uint32_t v) { return (uint32_t)__shfl_xor_sync(0xffffffffu, (int)v, 1); }
__device__ __forceinline__ double shfl_xor_d(double v) { return __shfl_xor_sync(0xffffffffu, v, 1); }

// Half h of the state's lanes as sums and differences of lanes i and i + 6.
__device__ __forceinline__ void duo_inputs(const uint64_t s[6], uint32_t h, double u[6], double w[6]) {
#pragma unroll
    for (int i = 0; i < 6; i++) {
        const uint32_t lo = (uint32_t)s[i], hi = (uint32_t)(s[i] >> 32);
        const uint32_t got = shfl_xor32(h ? lo : hi);  // the partner wants the half it computes
        const uint32_t mine = h ? hi : lo;
        const uint32_t a = h ? got : mine, b = h ? mine : got;  // lanes 0-5 are thread 0's, 6-11 thread 1's
        u[i] = sum_dbl(a, b);
        w[i] = diff_dbl(a, b);
    }
}
// Thread 0 keeps the low outputs of lanes 0-5 and receives their high outputs;
// thread 1 keeps the high outputs of lanes 6-11 and receives their low outputs.
__device__ __forceinline__ void duo_outputs(uint64_t s[6], uint32_t h, const double o[12]) {
#pragma unroll
    for (int i = 0; i < 6; i++) {
        const double got = shfl_xor_d(h ? o[i] : o[i + 6]);
        const double lo = h ? got : o[i], hi = h ? o[i + 6] : got;
        s[i] = pr_reduce_split(dbl_int(lo), dbl_int(hi));
    }
}
template <int N>
__device__ __forceinline__ void duo_rows(const double u[6], const double w[6], double o[12], const uint64_t *k) {
    using C = PoseidonCirc;
#pragma unroll
    for (int r = 0; r < 6; r++) {
        double pa = (double)C::p<N>(r, 5) * u[5], qa = (double)C::q<N>(r, 5) * w[5];
#pragma unroll
        for (int c = 4; c >= 0; c--) {
            pa = fma((double)C::p<N>(r, c), u[c], pa);
            qa = fma((double)C::q<N>(r, c), w[c], qa);
        }
        o[r] = fma(0.5, pa + qa, int_dbl(k[r]));
        o[r + 6] = fma(0.5, pa - qa, int_dbl(k[r + 6]));
    }
}

// s: lanes 6h .. 6h + 5 (partially reduced, in and out).  Every lane of the
// warp must call this (shuffles over the full warp).
__device__ __forceinline__ void poseidon_permute_duo(uint64_t s[6], uint32_t h, const PoseidonGroupTab &tab) {
    using C = PoseidonCirc;
    constexpr double d0 = (double)PoseidonMds::d0();
#pragma unroll
    for (int i = 0; i < 6; i++) s[i] = pr_add_c(s[i], tab.rc0[6 * h + i]);
#pragma unroll 1
    for (int half = 0; half < 2; half++) {
#pragma unroll 1
        for (int f = 0; f < 4; f++) {
#pragma unroll
            for (int i = 0; i < 6; i++) s[i] = pr_pow7<true>(s[i]);
            double u[6], w[6], o[12];
            duo_inputs(s, h, u, w);
            duo_rows<1>(u, w, o, tab.full[4 * half + f][h]);
            // x0 is (u + w - 2^32) / 2; both are exact
            o[0] = fma(0.5 * d0, u[0] + (w[0] - int_dbl(1ull << 32)), o[0]);
            duo_outputs(s, h, o);
        }
        if (half) break;
#pragma unroll 1
        for (int q = 0; q < 11; q++) {
            if (h == 0) s[0] = pr_pow7<true>(s[0]);
            double u[6], w[6], o[12];
            duo_inputs(s, h, u, w);
            const double x0 = 0.5 * (u[0] + (w[0] - int_dbl(1ull << 32)));
            double pa = 0, qa = 0;
#pragma unroll
            for (int i = 5; i >= 0; i--) {
                pa = fma((double)C::p<1>(0, i), u[i], pa);
                qa = fma((double)C::q<1>(0, i), w[i], qa);
            }
            const double y0 = fma(0.5, pa + qa, fma(d0, x0, int_dbl(tab.mid[q][h])));
            const double other = shfl_xor_d(y0);
            const uint64_t y = pr_pow7<true>(pr_reduce_split(dbl_int(h ? other : y0), dbl_int(h ? y0 : other)));
            const double yp = word_dbl(h ? (uint32_t)(y >> 32) : (uint32_t)y);
            const double g = fma(d0, x0, yp - y0);
            duo_rows<2>(u, w, o, tab.pair[q][h]);
#pragma unroll
            for (int r = 0; r < 12; r++) o[r] = fma((double)C::at(-r), g, o[r]);
            o[0] = fma(d0, yp, o[0]);
            duo_outputs(s, h, o);
        }
    }
}

// Sponge of n words on a lane pair (zeknox's hash_or_noop: n <= 4 copies and
// zero-pads); `active` pairs load and store, the others compute on zeros.
// n must be the same for all pairs of a warp.
__device__ __forceinline__ void poseidon_hash_one_duo(const uint64_t *in, uint32_t n, uint64_t *out, bool active,
                                                      uint32_t h, const PoseidonGroupTab &tab) {
    if (n <= 4) {
        if (active && h == 0)
            for (uint32_t i = 0; i < 4; i++) out[i] = i < n ? in[i] : 0ull;
        return;
    }
    uint64_t s[6] = {0, 0, 0, 0, 0, 0};
    for (uint32_t idx = 0; idx < n; idx += 8) {
        const uint32_t len = n - idx < 8 ? n - idx : 8;
        if (active) {
#pragma unroll
            for (uint32_t i = 0; i < 6; i++) {
                const uint32_t lane = 6 * h + i;  // rate lanes 0..7 are overwritten
                if (lane < len) s[i] = gl_canon(in[idx + lane]);
            }
        }
        poseidon_permute_duo(s, h, tab);
    }
    if (active && h == 0)
#pragma unroll
        for (int i = 0; i < 4; i++) out[i] = gl_canon(s[i]);
}

// ------------------------------------------- Poseidon on six threads
// For the latency-bound parts (narrow tree levels, small trees) one
// permutation is spread over a group of six consecutive lanes of a warp
// (five groups per warp; lanes 30 and 31 compute on dummy data).  Group
// thread t owns lanes t and t + 6.  Each round or pair of partial rounds: an
// all-gather of the 12 lanes by shuffles (every shuffle reads one thread of
// the group, so all threads get the lanes in natural order), then thread t
// computes the row pair (t, t + 6) of the layer, its rows of A + B and A - B
// held in registers.  Full rounds apply the S-box to the owned lanes before
// the gather; in a pair every thread runs both of lane 0's S-boxes itself, so
// that a pair needs one gather and no further exchange, and the other lanes'
// shuffles hide behind the first S-box.
struct HexLanes {
    uint32_t t;     // thread within the group, 0..5 (lanes 30, 31: 0..1 of a dummy group)
    uint32_t base;  // warp lane of the group's thread 0
    __device__ __forceinline__ HexLanes() {
        const uint32_t lane = threadIdx.x & 31;
        const uint32_t g = lane < 30 ? lane / 6 : 0;
        t = lane < 30 ? lane % 6 : lane - 30;
        base = 6 * g;
    }
    // true for the lanes whose group is a real one (not lanes 30, 31)
    __device__ __forceinline__ bool real() const { return (threadIdx.x & 31) < 30; }
    __device__ __forceinline__ uint32_t group_in_warp() const { return base / 6; }
};
// Poseidon's group: its rows in registers.
struct HexGroup : HexLanes {
    double p1[6], q1[6];  // row t of A + B and A - B
    double p2[6], q2[6];  // row t of their squares
    double c0, c6;        // C e0 at rows t and t + 6
    double d0;            // the diagonal term on thread 0, else 0
    __device__ __forceinline__ explicit HexGroup(const PoseidonGroupTab &tab) : HexLanes() {
        const double *row = tab.rows[t];
#pragma unroll
        for (int k = 0; k < 6; k++) {
            p1[k] = row[k];
            q1[k] = row[6 + k];
            p2[k] = row[12 + k];
            q2[k] = row[18 + k];
        }
        c0 = row[24];
        c6 = row[25];
        d0 = t == 0 ? (double)PoseidonMds::d0() : 0.0;
    }
};

__device__ __forceinline__ uint64_t shfl64(uint64_t v, uint32_t src) {
    return (uint64_t)__shfl_sync(0xffffffffu, (long long)v, (int)src);
}

// o0, o1: lanes t and t + 6 of the state (partially reduced, in and out).
// Every lane of the warp must call this (shuffles over the full warp).
__device__ __forceinline__ void poseidon_permute_hex(uint64_t &o0, uint64_t &o1, const HexGroup &g,
                                                     const PoseidonGroupTab &tab) {
    using C = PoseidonCirc;
    constexpr double d0 = (double)PoseidonMds::d0();
    o0 = pr_add_c(o0, tab.rc0[g.t]);
    o1 = pr_add_c(o1, tab.rc0[g.t + 6]);
#pragma unroll 1
    for (int half = 0; half < 2; half++) {
#pragma unroll 1
        for (int f = 0; f < 4; f++) {
            o0 = pr_pow7(o0);
            o1 = pr_pow7(o1);
            uint64_t x[12];
#pragma unroll
            for (int i = 0; i < 12; i++) x[i] = shfl64(i < 6 ? o0 : o1, g.base + (i % 6));
            double first[2], second[2];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                double pa = 0, qa = 0;
#pragma unroll
                for (int k = 0; k < 6; k++) {
                    pa = fma(g.p1[k], sum_dbl(half_of(x[k], h), half_of(x[k + 6], h)), pa);
                    qa = fma(g.q1[k], diff_dbl(half_of(x[k], h), half_of(x[k + 6], h)), qa);
                }
                first[h] = fma(0.5, pa + qa,
                               fma(g.d0, word_dbl(half_of(x[0], h)), int_dbl(tab.full[4 * half + f][h][g.t])));
                second[h] = fma(0.5, pa - qa, int_dbl(tab.full[4 * half + f][h][g.t + 6]));
            }
            o0 = pr_reduce_split(dbl_int(first[0]), dbl_int(first[1]));
            o1 = pr_reduce_split(dbl_int(second[0]), dbl_int(second[1]));
        }
        if (half) break;
#pragma unroll 1
        for (int q = 0; q < 11; q++) {
            uint64_t x[12];
#pragma unroll
            for (int i = 0; i < 12; i++) x[i] = shfl64(i < 6 ? o0 : o1, g.base + (i % 6));
            x[0] = pr_pow7(x[0]);
            double first[2], second[2], y0[2];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                double pa = 0, qa = 0, pb = 0, qb = 0;
#pragma unroll
                for (int k = 5; k >= 0; k--) {
                    const double u = sum_dbl(half_of(x[k], h), half_of(x[k + 6], h));
                    const double w = diff_dbl(half_of(x[k], h), half_of(x[k + 6], h));
                    pa = fma((double)C::p<1>(0, k), u, pa);
                    qa = fma((double)C::q<1>(0, k), w, qa);
                    pb = fma(g.p2[k], u, pb);
                    qb = fma(g.q2[k], w, qb);
                }
                y0[h] = fma(0.5, pa + qa, fma(d0, word_dbl(half_of(x[0], h)), int_dbl(tab.mid[q][h])));
                first[h] = fma(0.5, pb + qb, int_dbl(tab.pair[q][h][g.t]));
                second[h] = fma(0.5, pb - qb, int_dbl(tab.pair[q][h][g.t + 6]));
            }
            const uint64_t y = pr_pow7(pr_reduce_split(dbl_int(y0[0]), dbl_int(y0[1])));
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const double yp = word_dbl(half_of(y, h));
                const double e = fma(d0, word_dbl(half_of(x[0], h)), yp - y0[h]);
                first[h] = fma(g.d0, yp, fma(g.c0, e, first[h]));
                second[h] = fma(g.c6, e, second[h]);
            }
            o0 = pr_reduce_split(dbl_int(first[0]), dbl_int(first[1]));
            o1 = pr_reduce_split(dbl_int(second[0]), dbl_int(second[1]));
        }
    }
}

// ------------------------------------------- Poseidon2 on six threads
// The same group layout: thread t owns state lanes t and t + 6.
//
// External layer: output lane r is sum_b (1 + [b == r / 4]) (M4 x_b)[r % 4]
// over the three 4-lane blocks x_b.  Row c + 2 of M4 is row c rotated by two
// columns (M4[c + 2][d] = M4[c][d + 2], indices mod 4), and lane t + 6 has
// column (t + 2) % 4, so thread t needs only m = M4[t % 4]: lane t takes
// x_(4b + d) with m[d], lane t + 6 with m[(d + 2) % 4], and each lane weighs
// the three block sums by w in {1, 2}.  As in the one-thread layer, each
// 32-bit half runs in exact FP64 (every sum below 2^39).
//
// Internal layer (x_i <- x_i D_i + sum_j x_j + c_i): each thread adds its
// two lanes exactly (65 bits), the group all-gathers the six partial sums
// (96-bit total), and each thread forms its two lanes' products.
struct HexGroup2 : HexLanes {
    double m[4];          // row t % 4 of M4
    double w0[3], w1[3];  // block weights of lanes t and t + 6
    uint64_t d0, d1;      // internal diagonal of lanes t and t + 6, times 2^64
    __device__ __forceinline__ explicit HexGroup2(const Poseidon2Tab &tab) : HexLanes() {
        // M4 rows 0 and 1; rows 2 and 3 are these rotated by two columns.
        const uint32_t c = t & 3, r = c & 1, rot = c & 2;
#pragma unroll
        for (int d = 0; d < 4; d++) {
            const uint32_t k = (d + rot) & 3;
            const double row0 = k == 0 ? 5.0 : k == 1 ? 7.0 : k == 2 ? 1.0 : 3.0;
            const double row1 = k == 0 ? 4.0 : k == 1 ? 6.0 : 1.0;
            m[d] = r ? row1 : row0;
        }
#pragma unroll
        for (uint32_t b = 0; b < 3; b++) {
            w0[b] = b == t / 4 ? 2.0 : 1.0;
            w1[b] = b == (t + 6) / 4 ? 2.0 : 1.0;
        }
        d0 = tab.diag[t];
        d1 = tab.diag[t + 6];
    }
};

// External layer on a group, plus the constants c.
__device__ __forceinline__ void poseidon2_external_hex(uint64_t &o0, uint64_t &o1, const HexGroup2 &g,
                                                       const uint64_t *c) {
    uint64_t x[12];
#pragma unroll
    for (int i = 0; i < 12; i++) x[i] = shfl64(i < 6 ? o0 : o1, g.base + (i % 6));
    double first[2], second[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        double v[12];
#pragma unroll
        for (int i = 0; i < 12; i++) v[i] = word_dbl(half_of(x[i], h));
        double a0 = 0, a1 = 0;
#pragma unroll
        for (int b = 0; b < 3; b++) {
            double y0 = g.m[0] * v[4 * b], y1 = g.m[2] * v[4 * b];
#pragma unroll
            for (int d = 1; d < 4; d++) {
                y0 = fma(g.m[d], v[4 * b + d], y0);
                y1 = fma(g.m[(d + 2) & 3], v[4 * b + d], y1);
            }
            a0 = fma(g.w0[b], y0, a0);
            a1 = fma(g.w1[b], y1, a1);
        }
        first[h] = a0;
        second[h] = a1;
    }
    o0 = pr_reduce_split_add(dbl_int(first[0]), dbl_int(first[1]), c[g.t]);
    o1 = pr_reduce_split_add(dbl_int(second[0]), dbl_int(second[1]), c[g.t + 6]);
}

// Internal layer on a group (poseidon2_internal without the constant).
__device__ __forceinline__ void poseidon2_internal_hex(uint64_t &o0, uint64_t &o1, const HexGroup2 &g) {
    uint32_t p0, p1, p2;
    asm("add.cc.u32 %0, %3, %5;\n\t"
        "addc.cc.u32 %1, %4, %6;\n\t"
        "addc.u32 %2, 0, 0;"
        : "=r"(p0), "=r"(p1), "=r"(p2)
        : "r"((uint32_t)o0), "r"((uint32_t)(o0 >> 32)), "r"((uint32_t)o1), "r"((uint32_t)(o1 >> 32)));
    uint32_t s0 = 0, s1 = 0, s2 = 0;  // sum of the 12 lanes, below 12 * 2^64
#pragma unroll
    for (int k = 0; k < 6; k++) {
        const uint32_t src = g.base + k;
        const uint32_t q0 = (uint32_t)__shfl_sync(0xffffffffu, (int)p0, (int)src);
        const uint32_t q1 = (uint32_t)__shfl_sync(0xffffffffu, (int)p1, (int)src);
        const uint32_t q2 = (uint32_t)__shfl_sync(0xffffffffu, (int)p2, (int)src);
        asm("add.cc.u32 %0, %0, %3;\n\t"
            "addc.cc.u32 %1, %1, %4;\n\t"
            "addc.u32 %2, %2, %5;"
            : "+r"(s0), "+r"(s1), "+r"(s2)
            : "r"(q0), "r"(q1), "r"(q2));
    }
    const uint64_t sum = poseidon2_sum_mont(s0, s1, s2);
    o0 = poseidon2_lane(o0, g.d0, sum);
    o1 = poseidon2_lane(o1, g.d1, sum);
}

// The rounds of poseidon2_permute on a group.
__device__ __forceinline__ void poseidon2_permute_hex(uint64_t &o0, uint64_t &o1, const HexGroup2 &g,
                                                      const Poseidon2Tab &tab) {
    poseidon2_external_hex(o0, o1, g, tab.rc[0]);
#pragma unroll 1
    for (int half = 0; half < 2; half++) {
#pragma unroll 1
        for (int f = 0; f < 4; f++) {
            o0 = pr_pow7(o0);
            o1 = pr_pow7(o1);
            poseidon2_external_hex(o0, o1, g, tab.rc[26 * half + f + 1]);
        }
        if (half) break;
#pragma unroll 1
        for (int rnd = 4; rnd < 26; rnd++) {
            const uint64_t y = pr_pow7(o0);
            if (g.t == 0) o0 = y;
            poseidon2_internal_hex(o0, o1, g);
            o0 = pr_add_c(o0, tab.rc[rnd + 1][g.t]);  // only lane 0's is non-zero before round 26
            if (rnd == 25) o1 = pr_add_c(o1, tab.rc[26][g.t + 6]);
        }
    }
}

__device__ __forceinline__ void permute_hex(uint64_t &o0, uint64_t &o1, const HexGroup &g, const PoseidonGroupTab &tab) {
    poseidon_permute_hex(o0, o1, g, tab);
}
__device__ __forceinline__ void permute_hex(uint64_t &o0, uint64_t &o1, const HexGroup2 &g, const Poseidon2Tab &tab) {
    poseidon2_permute_hex(o0, o1, g, tab);
}

// The group form of a hasher: HexOf<kPoseidon> or HexOf<kPoseidon2>.
template <int H>
using HexOf = typename std::conditional<H == kPoseidon, HexGroup, HexGroup2>::type;

// H(l || r) on a group: every lane calls; `active` groups load and store.
template <class G, class Tab>
__device__ __forceinline__ void hash_two_hex(const uint64_t *l, const uint64_t *r, uint64_t *out, bool active,
                                             const G &g, const Tab &tab) {
    uint64_t o0 = 0, o1 = 0;
    if (active) {
        o0 = gl_canon(g.t < 4 ? l[g.t] : r[g.t - 4]);
        if (g.t < 2) o1 = gl_canon(r[g.t + 2]);
    }
    permute_hex(o0, o1, g, tab);
    if (active && g.t < 4) out[g.t] = gl_canon(o0);
}

// Sponge of n words (zeknox's hash_or_noop: n <= 4 copies and zero-pads).
// n must be the same for all groups of a warp.
template <class G, class Tab>
__device__ __forceinline__ void hash_one_hex(const uint64_t *in, uint32_t n, uint64_t *out, bool active, const G &g,
                                             const Tab &tab) {
    if (n <= 4) {
        if (active && g.t < 4) out[g.t] = g.t < n ? in[g.t] : 0ull;
        return;
    }
    uint64_t o0 = 0, o1 = 0;
    for (uint32_t idx = 0; idx < n; idx += 8) {
        const uint32_t len = n - idx < 8 ? n - idx : 8;
        if (active) {
            if (g.t < len) o0 = gl_canon(in[idx + g.t]);
            if (g.t + 6 < len) o1 = gl_canon(in[idx + g.t + 6]);
        }
        permute_hex(o0, o1, g, tab);
    }
    if (active && g.t < 4) out[g.t] = gl_canon(o0);
}

// --------------------------------------- Poseidon-BN128 on five threads
// One thread's permutation is ~130,000 wide multiplies, so a tree of a few
// thousand leaves, or a narrow level, leaves most of the GPU idle and waits for
// one thread.  Here a group of five consecutive lanes (six groups per warp,
// lanes 30 and 31 on dummy data) takes one hash, thread t owning state lane t.
// Full rounds: each thread its lane's S-box, a gather of the five lanes, and
// its row of the matrix.  Partial rounds: lane 0 is kept by every thread, which
// all run its S-box; each thread forms its term of the row sum and, for t > 0,
// its lane's update; the terms are summed by shuffles.  2.5 times the multiplies
// of the one-thread form in all, and 0.4 times per thread.
struct BnLanes {
    uint32_t t, base;  // thread within the group, warp lane of the group's thread 0
    __device__ __forceinline__ BnLanes() {
        const uint32_t lane = threadIdx.x & 31, l = lane < 30 ? lane : lane - 30;
        t = l % 5;
        base = l - t;
    }
    __device__ __forceinline__ bool real() const { return (threadIdx.x & 31) < 30; }
    __device__ __forceinline__ uint32_t group_in_warp() const { return base / 5; }
};
__device__ __forceinline__ Fr bn_shfl(const Fr &x, uint32_t src) {
    Fr y;
#pragma unroll
    for (int l = 0; l < kBnL; l++) y.v[l] = __shfl_sync(0xffffffffu, x.v[l], (int)src);
    return y;
}

// lane: the three words of lanes 3 (t - 1) .. 3 (t - 1) + 2 on thread t > 0.
// Every lane of the warp must call this.
__device__ __forceinline__ void bn_permute_group(uint64_t lane[3], const BnLanes &g, const BnTab &tab) {
    Fr x = bn_from_words(lane, tab.c[g.t], tab);
    if (g.t == 0) x = tab.c[0];
#pragma unroll 1
    for (int half = 0; half < 2; half++) {
#pragma unroll 1
        for (int r = 0; r < 4; r++) {
            Fr k{};
            if (!half) k = tab.c[5 * (r + 1) + g.t];
            else if (r < 3) k = tab.c[85 + 5 * r + g.t];
            x = bn_sbox_add(x, k);
            const Fr *m = !half && r == 3 ? tab.p : tab.m;
            BnCols t = bn_zero();
#pragma unroll 1
            for (uint32_t j = 0; j < 5; j++) bn_acc(t, bn_shfl(x, g.base + j), m[5 * j + g.t]);
            x = bn_reduce(t);
        }
        if (half) break;
        Fr z = bn_shfl(x, g.base);  // lane 0
#pragma unroll 1
        for (int r = 0; r < 60; r++) {
            const Fr *sp = tab.s + 9 * r;
            z = bn_sbox_add(z, tab.c[25 + r]);
            Fr a;
#pragma unroll
            for (int l = 0; l < kBnL; l++) a.v[l] = g.t == 0 ? z.v[l] : x.v[l];
            BnCols u = bn_addend(x), t = bn_zero();
            bn_acc(t, a, sp[g.t]);
            bn_acc(u, z, sp[4 + g.t]);  // thread 0's is not used
            const Fr y = bn_reduce(t);
            x = bn_reduce(u);
            uint32_t carry = 0;
#pragma unroll
            for (int l = 0; l < kBnL; l++) {  // the sum of the five terms, limbs below 2^29 again
                uint32_t v = carry;
#pragma unroll
                for (uint32_t j = 0; j < 5; j++) v += __shfl_sync(0xffffffffu, y.v[l], (int)(g.base + j));
                z.v[l] = v & kBnMask;
                carry = v >> 29;
            }
        }
        if (g.t == 0) x = z;
    }
    uint64_t w[3];
    bn_words(x, w);  // state lane i gives words 3 i .. 3 i + 2, which thread i + 1 takes on
#pragma unroll
    for (int k = 0; k < 3; k++) lane[k] = shfl64(w[k], g.t ? g.base + g.t - 1 : g.base);
}

// The sponge (n <= 4 copies and zero-pads) and H(l || r) on a group; `active`
// groups load and store.  n must be the same for all groups of a warp.
__device__ __forceinline__ void bn_store(const uint64_t lane[3], uint64_t *out, const BnLanes &g) {
    if (g.t == 1) {
        out[0] = lane[0];
        out[1] = lane[1];
        out[2] = lane[2];
    }
    if (g.t == 2) out[3] = lane[0];
}
__device__ __forceinline__ void bn_hash_one_group(const uint64_t *in, uint32_t n, uint64_t *out, bool active,
                                                  const BnLanes &g, const BnTab &tab) {
    if (n <= 4) {
        if (active && g.t < 4) out[g.t] = g.t < n ? in[g.t] : 0ull;
        return;
    }
    uint64_t lane[3] = {0, 0, 0};
#pragma unroll 1
    for (uint32_t idx = 0; idx < n; idx += 8) {
        const uint32_t len = n - idx < 8 ? n - idx : 8;
        if (active && g.t > 0) {
#pragma unroll
            for (uint32_t k = 0; k < 3; k++)
                if (3 * (g.t - 1) + k < len) lane[k] = gl_canon(in[idx + 3 * (g.t - 1) + k]);
        }
        bn_permute_group(lane, g, tab);
    }
    if (active) bn_store(lane, out, g);
}
__device__ __forceinline__ void bn_hash_two_group(const uint64_t *l, const uint64_t *r, uint64_t *out, bool active,
                                                  const BnLanes &g, const BnTab &tab) {
    uint64_t lane[3] = {0, 0, 0};
    if (active && g.t > 0) {
#pragma unroll
        for (uint32_t k = 0; k < 3; k++) {
            const uint32_t i = 3 * (g.t - 1) + k;
            if (i < 8) lane[k] = gl_canon(i < 4 ? l[i] : r[i - 4]);
        }
    }
    bn_permute_group(lane, g, tab);
    if (active) bn_store(lane, out, g);
}

}  // namespace zk
