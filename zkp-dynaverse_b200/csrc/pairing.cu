// BN254 optimal ate pairing and pairing-product checks on sm_100a.
//
// The verifier's checks (crates/protocol/src/verification.rs:37-144):
// PairingChecks::equal / equal_prepared / product_equal reduce one equation
// to prod_k e(P_k, Q_k) = 1 (right-hand G1 points negated by the caller),
// computed by Bn254::multi_miller_loop and final_exponentiation.  Here a
// launch takes many equations: a group of lanes runs the Miller loop of
// one term (or, with prepared G2 points in large batches, the multi-Miller
// loop of one equation), then a group per equation multiplies its terms'
// values and runs the final exponentiation.  The reference's native Miller probe
// (native/include/dynaverse_bn254_miller.h) is a diagnostic of line traces
// and is not reproduced.
//
// Fq12 = Fq2[w]/(w^6 - xi), xi = 9 + u, held by twelve lanes, one component
// each (see "lane groups"): products, squares and the sparse line product
// c_k = sum_i f_i l_(k-i) are sums of base products per lane with one
// reduction; the q-power Frobenius is conj(a_k) xi^(k(q-1)/6) per lane;
// f^(q^6) negates the odd coefficients.  The
// serialised GT element uses the tower Fq12 = Fq6[w]/(w^2 - v), Fq6 =
// Fq2[v]/(v^3 - xi), v = w^2: c0 = (w^0, w^2, w^4), c1 = (w^1, w^3, w^5).
//
// Miller loop over the NAF of 6z + 2 (z the BN seed), then the lines to
// pi(Q) and -pi^2(Q).  T is kept in Jacobian coordinates on the twist
// E': y^2 = x^3 + 3/xi, untwisted by (x, y) -> (x w^2, y w^3).  The line
// through T (slope lam) at P = (xp, yp) is yp - lam xp w + (lam xT - yT) w^3;
// each step multiplies it by a nonzero Fq2 factor (killed by the final
// exponentiation, since Fq2* lies in the kernel of q^6 - 1).  The products
// of a step are spread over the group's lanes level by level:
//   doubling, x = X/Z^2, y = Y/Z^3, factor 2 Y Z^3:
//     (2 Y Z^3 yp) + (-3 X^2 Z^2 xp) w + (3 X^3 - 2 Y^2) w^3
//   addition of affine S = (xs, ys), H = xs Z^2 - X, R = ys Z^3 - Y, factor 2 Z H:
//     (2 Z H yp) + (-2 R xp) w + (2 R xs - 2 Z H ys) w^3
// with the doubling and mixed-addition formulas dbl-2009-l and
// madd-2007-bl (Explicit-Formulas Database) for the point itself.
//
// Final exponentiation: the easy part (q^6 - 1)(q^2 + 1) by conjugation,
// inversion and a q^2 Frobenius, then the exponent
// 2z(6z^2 + 3z + 1)(q^4 - q^2 + 1)/r, whose base-q digits are
//   l0 = 12z^3 + 12z^2 + 6z + 1, l1 = 12z^3 + 6z^2 + 4z,
//   l2 = 12z^3 + 6z^2 + 6z,      l3 = 12z^3 + 6z^2 + 4z - 1
// (Fuentes-Castaneda, Knapp and Rodriguez-Henriquez, "Faster hashing to
// G2", SAC 2011), from a = f^z, b = a^z, c = b^z:
//   T = c^12 b^6, f^l1 = T a^4, f^l2 = T a^6, f^l3 = f^l1 conj(f),
//   f^l0 = c^12 b^12 a^6 f, result = f^l0 (f^l1)^q (f^l2)^(q^2) (f^l3)^(q^3).
// conj is the inverse after the easy part (the result is in the
// cyclotomic subgroup, where squares take the Granger-Scott form); the easy part's inverse is conj(f) / N with N =
// f conj(f) in Fq6 inverted in every lane.  A verdict is result == 1; the
// value written for a single pairing is the GT element in the tower order
// above, canonical.
#include <cstring>
#include <map>
#include <memory>
#include <unordered_map>
#include <string>
#include <vector>

#include "abi_util.hpp"
#include "backend.hpp"
#include "engine.hpp"

namespace dv {
namespace {

struct Fq6 {
    Fq2 c0, c1, c2;
};

// xi^(j (q-1)/6), j = 0..5, Montgomery (c0, c1).
__device__ __constant__ uint32_t FROB1[6][2][8] = {
    {{0xc58f0d9du, 0xd35d438du, 0xf5c70b3du, 0x0a78eb28u, 0x7879462cu, 0x666ea36fu, 0x9a07df2fu, 0x0e0a77c1u},
     {0x00000000u, 0x00000000u, 0x00000000u, 0x00000000u, 0x00000000u, 0x00000000u, 0x00000000u, 0x00000000u}},
    {{0x33144907u, 0xaf9ba696u, 0x87afb78au, 0xca6b1d73u, 0xf08a2087u, 0x11bded5eu, 0x1a1f3a7cu, 0x02f34d75u},
     {0x4c492d72u, 0xa222ae23u, 0x565de15bu, 0xd00f02a4u, 0x53dfc926u, 0xdc2ff3a2u, 0xb3899551u, 0x10a75716u}},
    {{0x4563ab30u, 0xb5773b10u, 0xa9aa6454u, 0x347f91c8u, 0x242e0991u, 0x7a007127u, 0x118214ecu, 0x1956bcd8u},
     {0xa0aa4757u, 0x6e849f1eu, 0x89f89141u, 0xaa1c7b6du, 0xfae0ca3au, 0xb6e713cdu, 0x4e82ebc3u, 0x26694fbbu}},
    {{0x2936b629u, 0xe4bbdd0cu, 0xe133bacbu, 0xbb30f162u, 0xf9645366u, 0x31a9d1b6u, 0xa500f8ddu, 0x253570beu},
     {0x5ffe77c7u, 0xa1d77ce4u, 0x7826d1dbu, 0x07affd11u, 0xbb7edc6bu, 0x6d16bd27u, 0x85defeccu, 0x2c872002u}},
    {{0x843abe92u, 0x7361d77fu, 0x273411fbu, 0xa5bb2bd3u, 0x4b3e2399u, 0x9c941f31u, 0xbb9fd3ecu, 0x15df9cddu},
     {0x4bd8c949u, 0x5dddfd15u, 0xa4445b60u, 0x62cb29a5u, 0x0c7dd2b9u, 0x37bc870au, 0x3171f0fdu, 0x24830a9du}},
    {{0x41690fe7u, 0xc970692fu, 0x27694b0bu, 0xe2403421u, 0x83c459e8u, 0x32bee66bu, 0x0ab08841u, 0x12aabcedu},
     {0x40aebfa9u, 0x0d485d23u, 0xab2fcc57u, 0x05193418u, 0x8a4910f5u, 0xd3b0a40bu, 0x35d2925au, 0x2f21ebb5u}}};
// |xi^(j (q-1)/6)|^2 = xi^(j (q^2-1)/6) in Fq, Montgomery.
__device__ __constant__ uint32_t FROB2[6][8] = {
    {0xc58f0d9du, 0xd35d438du, 0xf5c70b3du, 0x0a78eb28u, 0x7879462cu, 0x666ea36fu, 0x9a07df2fu, 0x0e0a77c1u},
    {0x00fa1bf2u, 0xca8d8005u, 0x68b39769u, 0xf0c5d614u, 0xad0d4418u, 0x0e201271u, 0xbad856e6u, 0x04290f65u},
    {0x13e80b9cu, 0x3350c88eu, 0xdb5e56b9u, 0x7dce557cu, 0xb615564au, 0x6001b4b8u, 0x020217e0u, 0x2682e617u},
    {0x12edefaau, 0x68c34889u, 0x72aabf4fu, 0x8d087f68u, 0x09081231u, 0x51e1a247u, 0x4729c0fau, 0x2259d6b1u},
    {0xd782e155u, 0x71930c11u, 0xffbe3323u, 0xa6bb947cu, 0xd4741444u, 0xaa303344u, 0x26594943u, 0x2c3b3f0du},
    {0xc494f1abu, 0x08cfc388u, 0x8d1373d4u, 0x19b31514u, 0xcb6c0213u, 0x584e90fdu, 0xdf2f8849u, 0x09e1685bu}};
// NAF of 6z + 2, most significant digit first.
__device__ __constant__ int8_t NAF_6Z2[66] = {1, 0, -1, 0, 1, 0, 0, 0, -1, 0, -1, 0, 0, 0, -1, 0, 1, 0, -1, 0, 0, -1, 0, 0, 0, 0, 0, 1, 0, 0, -1, 0, 1, 0, 0, -1, 0, 0, 0, 0, -1, 0, 1, 0, 0, 0, -1, 0, -1, 0, 0, 1, 0, 0, 0, -1, 0, 0, -1, 0, 1, 0, 1, 0, 0, 0};
constexpr int NAF_LEN = 66;
// Width-4 NAF of z, most significant digit first: 14 odd digits in
// {+-1, +-3, +-5, +-7} (against 24 in the plain NAF and 28 binary).
__device__ __constant__ int8_t WNAF_Z[63] = {1, 0, 0, 0, 0, 0, 5, 0, 0, 0, 0, -3, 0, 0, 0, 3, 0, 0, 0, 0, 5, 0, 0, 0, -5, 0, 0, 0, -3, 0, 0, 0, 1, 0, 0, 0, 0, 5, 0, 0, 0, 0, 7, 0, 0, 0, -7, 0, 0, 0, 0, 0, 0, 5, 0, 0, 0, 0, -1, 0, 0, 0, 1};
constexpr int WNAF_Z_LEN = 63;

DV_INL Fq load_fq(const uint32_t* w) {
    Fq r;
#pragma unroll
    for (int i = 0; i < 8; ++i) r.v[i] = w[i];
    return r;
}
DV_INL Fq2 frob1(int j) { return {load_fq(FROB1[j][0]), load_fq(FROB1[j][1])}; }
DV_INL Fq frob2(int j) { return load_fq(FROB2[j]); }

DV_INL Fq mul9(const Fq& a) { return Fq::add(Fq::dbl(Fq::dbl(Fq::dbl(a))), a); }
// (a0 + a1 u)(9 + u) = (9 a0 - a1) + (a0 + 9 a1) u
DV_INL Fq2 mul_xi(const Fq2& a) { return {Fq::sub(mul9(a.c0), a.c1), Fq::add(a.c0, mul9(a.c1))}; }


// 1 / a in Fq6 (one Fq inversion).
__device__ __noinline__ Fq6 f6_inv(const Fq6& a) {
    const Fq2 t0 = Fq2::sub(Fq2::sqr(a.c0), mul_xi(Fq2::mul(a.c1, a.c2)));
    const Fq2 t1 = Fq2::sub(mul_xi(Fq2::sqr(a.c2)), Fq2::mul(a.c0, a.c1));
    const Fq2 t2 = Fq2::sub(Fq2::sqr(a.c1), Fq2::mul(a.c0, a.c2));
    const Fq2 d = Fq2::add(Fq2::mul(a.c0, t0), mul_xi(Fq2::add(Fq2::mul(a.c2, t1), Fq2::mul(a.c1, t2))));
    const Fq2 di = Fq2::inv(d);
    return {Fq2::mul(t0, di), Fq2::mul(t1, di), Fq2::mul(t2, di)};
}

// ------------------------------------------------------------------ lane groups
// One Fq12 lives in a group of 16 lanes, twelve of them at work: lane 2k + c
// holds component c of the Fq2 coefficient of w^k.  Lanes 12 to 15 run along
// as copies of lanes 0 to 3 and write nothing.  The operands of a product go
// through shared memory (A plain; B with xi B and the negated second
// components beside it), and every lane sums the products of its component at
// 512 bits and reduces once: schoolbook rows with one reduction are fewer
// multiply-adds a lane than Karatsuba products reduced one by one, and leave
// no additions between lanes.
//
// H = 2 gives a group the whole warp: lanes 16 to 31 take the products with
// the second components of A, and the two half sums meet in one shuffle.  A
// group then needs 456 multiply-adds a lane for a product against 840 with
// H = 1 and two groups a warp.  These kernels are chains of dependent
// products, so H = 2 is taken while a call's groups leave the GPU's warp
// slots free, H = 1 (a tenth less work a group) beyond that.
//
// Bounds: a sum of up to 12 products of residues is below 12 p^2 < 2^511; its
// reduction is below 3.3 p, with 2 p added beforehand 5.27 p, and 2^256 is
// 5.29 p.
constexpr unsigned FULL = 0xffffffffu;
constexpr int THREADS = 128;
template <int H>
constexpr int GROUPS_PER_BLOCK = THREADS / (16 * H);
// Shared memory in Fq units: the multiples 0..9 of q, then per group
// A (6 coefficients and a zero one), B (per coefficient: b0, b1, -b1 and the
// same of xi b) and V (the products of a level).
constexpr int SM_MULT = 10, SM_A = 0, SM_B = 14, SM_V = 50, SM_GROUP = 62;
template <int H>
constexpr size_t SM_BYTES = sizeof(Fq) * (SM_MULT + SM_GROUP * GROUPS_PER_BLOCK<H>);
extern __shared__ uint4 pairing_sm[];
DV_INL Fq* sm(int i) { return reinterpret_cast<Fq*>(pairing_sm) + i; }

struct Lane {
    int k, c, h, at;  // coefficient, component, half; the group's place in shared memory
    bool writes;      // not a copy
    uint64_t group;   // global group index
};
// Also fills the block's tables; ends with a block barrier.
template <int H>
DV_INL Lane lane_setup() {
    const int l = threadIdx.x & 31, j = l & 15, jj = j < 12 ? j : j - 12;
    const int slot = (int)(threadIdx.x >> 5) * (2 / H) + (H == 1 ? l >> 4 : 0);
    Lane g;
    g.k = jj >> 1;
    g.c = jj & 1;
    g.h = H == 2 ? l >> 4 : 0;
    g.at = SM_MULT + SM_GROUP * slot;
    g.writes = j < 12 && g.h == 0;
    g.group = (uint64_t)blockIdx.x * GROUPS_PER_BLOCK<H> + slot;
    if (threadIdx.x < SM_MULT) {
        Fq m = Fq::zero();
        for (int i = 0; i < (int)threadIdx.x; ++i) m = Fq::add_raw(m, Fq::modulus());
        *sm(threadIdx.x) = m;
    }
    if (j < 2) *sm(g.at + SM_A + 12 + j) = Fq::zero();
    __syncthreads();
    return g;
}
DV_INL Fq dbl_raw(const Fq& a, int by = 1) {
    Fq r;
    r.v[0] = a.v[0] << by;
#pragma unroll
    for (int w = 1; w < 8; ++w) r.v[w] = __funnelshift_l(a.v[w - 1], a.v[w], by);
    return r;
}
DV_INL Fq neg_raw(const Fq& a) { return Fq::sub_raw(Fq::modulus(), a); }  // q - a (q for 0)
// v - (a multiple of q) in [0, q) for v < 10 q with top = v >> 252: the
// quotient 21 top / 64 is never too large and at most one too small.
DV_INL Fq reduce_top(const Fq& low, uint32_t top) {
    Fq r = Fq::sub_raw(low, *sm((int)((top * 21u) >> 6)));
    Fq::reduce_once(r.v);
    return r;
}
// This lane's component of xi b: 9 b0 - b1 and 9 b1 + b0.
DV_INL Fq xi_part(const Fq& b, int c) {
    const Fq other = shfl_xor(b, 1);
    const Fq q = c ? other : neg_raw(other);
    const Fq s = dbl_raw(b, 3);
    uint32_t top = b.v[7] >> 29;
    Fq r;
    asm("add.cc.u32 %0, %9, %17;\n\taddc.cc.u32 %1, %10, %18;\n\taddc.cc.u32 %2, %11, %19;\n\t"
        "addc.cc.u32 %3, %12, %20;\n\taddc.cc.u32 %4, %13, %21;\n\taddc.cc.u32 %5, %14, %22;\n\t"
        "addc.cc.u32 %6, %15, %23;\n\taddc.cc.u32 %7, %16, %24;\n\taddc.u32 %8, %8, 0;"
        : "=&r"(r.v[0]), "=&r"(r.v[1]), "=&r"(r.v[2]), "=&r"(r.v[3]), "=&r"(r.v[4]), "=&r"(r.v[5]), "=&r"(r.v[6]),
          "=&r"(r.v[7]), "+r"(top)
        : "r"(s.v[0]), "r"(s.v[1]), "r"(s.v[2]), "r"(s.v[3]), "r"(s.v[4]), "r"(s.v[5]), "r"(s.v[6]), "r"(s.v[7]),
          "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]), "r"(b.v[4]), "r"(b.v[5]), "r"(b.v[6]), "r"(b.v[7]));
    asm("add.cc.u32 %0, %0, %9;\n\taddc.cc.u32 %1, %1, %10;\n\taddc.cc.u32 %2, %2, %11;\n\t"
        "addc.cc.u32 %3, %3, %12;\n\taddc.cc.u32 %4, %4, %13;\n\taddc.cc.u32 %5, %5, %14;\n\t"
        "addc.cc.u32 %6, %6, %15;\n\taddc.cc.u32 %7, %7, %16;\n\taddc.u32 %8, %8, 0;"
        : "+r"(r.v[0]), "+r"(r.v[1]), "+r"(r.v[2]), "+r"(r.v[3]), "+r"(r.v[4]), "+r"(r.v[5]), "+r"(r.v[6]),
          "+r"(r.v[7]), "+r"(top)
        : "r"(q.v[0]), "r"(q.v[1]), "r"(q.v[2]), "r"(q.v[3]), "r"(q.v[4]), "r"(q.v[5]), "r"(q.v[6]), "r"(q.v[7]));
    return reduce_top(r, (top << 4) | (r.v[7] >> 28));
}
// Staging of this lane's components (a barrier must stand before, after the
// last reads, and one after, before the next).
DV_INL void put_a(const Lane& g, const Fq& a) {
    if (g.writes) *sm(g.at + SM_A + 2 * g.k + g.c) = a;
}
DV_INL void put_b(const Lane& g, const Fq& b, const Fq& xb) {
    if (!g.writes) return;
    Fq* s = sm(g.at + SM_B + 6 * g.k);
    s[g.c] = b;
    s[3 + g.c] = xb;
    if (g.c) {
        s[2] = neg_raw(b);
        s[5] = neg_raw(xb);
    }
}
DV_INL Fq::Wide wide_zero() {
    Fq::Wide r;
#pragma unroll
    for (int w = 0; w < 16; ++w) r.v[w] = 0;
    return r;
}
// The sum over both halves (H = 2).
template <int H>
DV_INL Fq::Wide whole_sum(const Fq::Wide& a) {
    if constexpr (H == 1) {
        return a;
    } else {
        Fq::Wide o;
#pragma unroll
        for (int w = 0; w < 16; ++w) o.v[w] = __shfl_xor_sync(FULL, a.v[w], 16);
        return Fq::wide_add(a, o);
    }
}
DV_INL Fq redc_large(const Fq::Wide& t) {
    const Fq r = Fq::redc_raw(t);
    return reduce_top(r, r.v[7] >> 28);
}
// This lane's component of A_i B_j (xi B_j with v): its part of the two
// base products added to acc.
template <int H>
DV_INL void term(Fq::Wide& acc, const Lane& g, const Fq* a, const Fq* b, int dbl) {
    const int second = g.c ? 0 : 2;  // b0 for component 1, -b1 for component 0
    if constexpr (H == 2) {
        acc = Fq::wide_add(acc, Fq::mul_wide(dbl_raw(a[g.h], dbl), b[g.h ? second : g.c]));
    } else {
        acc = Fq::wide_add(acc, Fq::mul_wide(dbl_raw(a[0], dbl), b[g.c]));
        acc = Fq::wide_add(acc, Fq::mul_wide(dbl_raw(a[1], dbl), b[second]));
    }
}
// The staged product A B (six terms), A B for A with the coefficients of a
// line (w^0, w^1, w^3: three terms), or the square of the element staged as
// both (pairs i <= j with i + j = k modulo 6, doubled unless i = j: four terms
// for even k, three for odd k).
enum DotKind { DOT_FULL, DOT_LINE, DOT_SQUARE };
template <int H, DotKind KIND>
__device__ __noinline__ Fq g_dot(Lane g) {
    Fq::Wide acc = wide_zero();
    constexpr int TERMS = KIND == DOT_FULL ? 6 : KIND == DOT_LINE ? 3 : 4;
#pragma unroll 1
    for (int t = 0; t < TERMS; ++t) {
        int i, j, xi, dbl = 0;
        if constexpr (KIND == DOT_SQUARE) {
            i = (g.k >> 1) - t;
            if (i < 0) i += 6;
            j = g.k - i;
            if (j < 0) j += 6;
            xi = i + j >= 6;
            dbl = i != j;
            if (t == 3 && (g.k & 1)) i = 6;  // the zero coefficient
        } else {
            i = KIND == DOT_LINE && t == 2 ? 3 : t;
            j = g.k - i;
            xi = j < 0;
            if (xi) j += 6;
        }
        term<H>(acc, g, sm(g.at + SM_A + 2 * i), sm(g.at + SM_B + 6 * j + 3 * xi), dbl);
    }
    return redc_large(whole_sum<H>(acc));
}
template <int H>
DV_INL Fq g_mul_staged(const Lane& g, const Fq& a, const Fq& b, const Fq& xb) {
    __syncwarp();
    put_a(g, a);
    put_b(g, b, xb);
    __syncwarp();
    return g_dot<H, DOT_FULL>(g);
}
template <int H>
DV_INL Fq g_mul(const Lane& g, const Fq& a, const Fq& b) {
    return g_mul_staged<H>(g, a, b, xi_part(b, g.c));
}
template <int H>
DV_INL Fq g_sqr(const Lane& g, const Fq& a) {
    const Fq xa = xi_part(a, g.c);
    __syncwarp();
    put_a(g, a);
    put_b(g, a, xa);
    __syncwarp();
    return g_dot<H, DOT_SQUARE>(g);
}
// f (l0 + l1 w + l3 w^3), this lane's component of the line on lanes k = 0, 1, 3.
template <int H>
DV_INL Fq g_mul_line(const Lane& g, const Fq& f, const Fq& line) {
    const Fq xf = xi_part(f, g.c);
    __syncwarp();
    put_a(g, line);
    put_b(g, f, xf);
    __syncwarp();
    return g_dot<H, DOT_LINE>(g);
}
// Square of an element of the cyclotomic subgroup (every value after the
// easy part of the final exponentiation), by Granger and Scott ("Faster
// squaring in the cyclotomic subgroup of sixth degree extensions", PKC
// 2010): with A_i = f_i + f_(i+3) t over Fq4 = Fq2[t]/(t^2 - xi), t = w^3,
//   f^2 = (3 A0^2 - 2 conj A0) + (3 t A2^2 + 2 conj A1) w + (3 A1^2 - 2 conj A2) w^2.
// A^2 = (a^2 + xi b^2) + 2 a b t for A = a + b t: lanes k = 0, 2, 4 sum
// a a + b (xi b), lanes 3, 5 sum 2 a b, lane 1 sums 2 a (xi b).  Three
// products a lane with H = 1 (a a by (a0 + a1)(a0 - a1) or 2 a0 a1), two
// with H = 2; three times the sum and the linear term join before the one reduction.
template <int H>
__device__ __noinline__ Fq g_cyc_sqr(Fq f, Lane g) {
    const Fq xf = xi_part(f, g.c);
    __syncwarp();
    put_a(g, f);
    put_b(g, f, xf);
    __syncwarp();
    const int m = g.k == 0 || g.k == 3 ? 0 : (g.k == 2 || g.k == 5 ? 1 : 2);
    const bool real = !(g.k & 1);
    const Fq* a = sm(g.at + SM_A + 2 * m);
    const Fq* a3 = sm(g.at + SM_A + 2 * (m + 3));
    const Fq* b = sm(g.at + SM_B + 6 * m);
    const Fq* b3 = sm(g.at + SM_B + 6 * (m + 3));
    const int second = g.c ? 0 : 2;
    Fq::Wide acc;
    if constexpr (H == 2) {
        const int sel = g.h ? second : g.c;
        const Fq x = real ? a[g.h] : dbl_raw(a[g.h]);
        acc = Fq::mul_wide(x, real ? b[sel] : b3[sel + (g.k == 1 ? 3 : 0)]);
        const Fq y = real ? a3[g.h] : Fq::zero();
        acc = Fq::wide_add(acc, Fq::mul_wide(y, b3[3 + sel]));
    } else {
        const Fq a0 = a[0], a1 = a[1];
        const int xi = real || g.k == 1 ? 3 : 0;
        acc = Fq::mul_wide(real ? a3[0] : dbl_raw(a0), b3[xi + g.c]);
        acc = Fq::wide_add(acc, Fq::mul_wide(real ? a3[1] : dbl_raw(a1), b3[xi + second]));
        const Fq u = !real ? Fq::zero() : g.c ? dbl_raw(a0) : Fq::add_raw(a0, a1);
        const Fq v = g.c ? a1 : Fq::sub(a0, a1);
        acc = Fq::wide_add(acc, Fq::mul_wide(u, v));
    }
    acc = whole_sum<H>(acc);
    acc = Fq::wide_add(acc, Fq::wide_add(acc, acc));
    const Fq l = dbl_raw(real ? neg_raw(f) : f);  // -+2 f, times 2^256
    Fq hi;
#pragma unroll
    for (int w = 0; w < 8; ++w) hi.v[w] = acc.v[8 + w];
    hi = Fq::add_raw(hi, l);
#pragma unroll
    for (int w = 0; w < 8; ++w) acc.v[8 + w] = hi.v[w];
    return redc_large(acc);
}
// f^(q^6): w -> -w.
DV_INL Fq g_conj(const Fq& f, int k) { return (k & 1) ? Fq::neg(f) : f; }
// q^e-power Frobenius, e = 1, 2, 3: conj(f_k) xi^(k (q^e - 1) / 6) (f_k itself for e = 2).
DV_INL Fq g_frob(const Lane& g, const Fq& f, int e) {
    if (e == 2) return Fq::mul(f, frob2(g.k));
    Fq2 s = frob1(g.k);
    if (e == 3) s = Fq2::mul_fq(s, frob2(g.k));
    const Fq o = shfl_xor(f, 1);
    // component 0: f0 s0 + f1 s1; component 1: f0 s1 - f1 s0
    return Fq::mul_sub(o, s.c1, f, g.c ? s.c0 : Fq::neg(s.c0));
}
// f^-1 = conj(f) / N, N = f conj(f) in Fq6 (the even coefficients, v = w^2).
template <int H>
__device__ __noinline__ Fq g_inv(Fq f, Lane g) {
    const Fq c = g_conj(f, g.k);
    const Fq n = g_mul<H>(g, f, c);
    __syncwarp();
    if (g.writes) *sm(g.at + SM_V + 2 * g.k + g.c) = n;
    __syncwarp();
    const Fq* v = sm(g.at + SM_V);
    const Fq6 ni = f6_inv({{v[0], v[1]}, {v[4], v[5]}, {v[8], v[9]}});
    const Fq2 t = g.k == 0 ? ni.c0 : (g.k == 2 ? ni.c1 : ni.c2);
    return g_mul<H>(g, c, (g.k & 1) ? Fq::zero() : g.c ? t.c1 : t.c0);
}
// a^z for a in the cyclotomic subgroup (a^-1 = conj a), z the BN seed, over
// its width-4 NAF: a, a^3, a^5, a^7 first (one square, three products), then
// 62 squares and 13 products.  xi times each table entry is kept beside it.
template <int H>
__device__ __noinline__ Fq g_pow_z(Fq a, Lane g) {
    Fq tab[4], xtab[4];
    tab[0] = a;
    const Fq a2 = g_cyc_sqr<H>(a, g), xa2 = xi_part(a2, g.c);
    xtab[0] = xi_part(a, g.c);
#pragma unroll 1
    for (int j = 1; j < 4; ++j) {
        tab[j] = g_mul_staged<H>(g, tab[j - 1], a2, xa2);
        xtab[j] = xi_part(tab[j], g.c);
    }
    Fq r = tab[WNAF_Z[0] >> 1];
#pragma unroll 1
    for (int i = 1; i < WNAF_Z_LEN; ++i) {
        r = g_cyc_sqr<H>(r, g);
        const int d = WNAF_Z[i];
        if (d) {
            const int e = (d < 0 ? -d : d) >> 1;
            const Fq t = tab[e], x = xtab[e];
            const bool flip = d < 0 && (g.k & 1);
            r = g_mul_staged<H>(g, r, flip ? Fq::neg(t) : t, flip ? Fq::neg(x) : x);
        }
    }
    return r;
}
DV_INL Fq g_one(const Lane& g) { return g.k == 0 && g.c == 0 ? Fq::one() : Fq::zero(); }

struct Tw {
    Fq x, y, z;  // this lane's components of a Jacobian point on the twist
};
DV_INL Fq pick(int k, const Fq& v0, const Fq& v1, const Fq& v2, const Fq& v3, const Fq& v4, const Fq& v5) {
    return k == 0 ? v0 : k == 1 ? v1 : k == 2 ? v2 : k == 3 ? v3 : k == 4 ? v4 : v5;
}
// Up to six Fq2 products of a dependency level, product k on the lanes of
// coefficient k; level_get reads this lane's component of product j.
template <int H>
__device__ __noinline__ void level(Fq a, Fq b, Lane g) {
    __syncwarp();
    if (g.writes) {
        *sm(g.at + SM_A + 2 * g.k + g.c) = a;
        Fq* s = sm(g.at + SM_B + 6 * g.k);
        s[g.c] = b;
        if (g.c) s[2] = neg_raw(b);
    }
    __syncwarp();
    Fq::Wide acc = wide_zero();
    term<H>(acc, g, sm(g.at + SM_A + 2 * g.k), sm(g.at + SM_B + 6 * g.k), 0);
    const Fq r = Fq::redc(whole_sum<H>(acc));
    if (g.writes) *sm(g.at + SM_V + 2 * g.k + g.c) = r;
    __syncwarp();
}
DV_INL Fq level_get(const Lane& g, int j) { return *sm(g.at + SM_V + 2 * j + g.c); }

// A line of the Miller loop at P = (xp, yp) is A yp + (B xp) w + C w^3 with
// A, B, C depending on Q alone (the doubling: A = 2 Y Z^3, B = -3 X^2 Z^2,
// C = 3 X^3 - 2 Y^2; the addition: A = 2 Z H, B = -2 R, C = 2 R xs - 2 Z H ys).
// Preparing Q records the LINES triples of its loop once -- arkworks'
// G2Prepared, which the reference caches per distinct G2 point
// (crates/protocol/src/verification.rs:105-126) -- so the loop of every term
// that shares Q only scales them by its P and multiplies them in.
struct __align__(16) Line {
    Fq2 a, b, c;
};
struct LinePart {
    Fq a, b, c;  // this lane's components
};
constexpr int LINES = 88;  // 65 doublings, 21 NAF additions (nonzero digits after the first), 2 Frobenius additions

// T <- 2T and its line, the products in three levels:
//   A = X^2, B = Y^2, ZZ = Z^2, YZ = Y Z;
//   C = B^2, (X + B)^2, E ZZ, Z3 ZZ, E X, E^2   (E = 3A, Z3 = 2 Y Z);
//   E (D - X3)                                  (D = 2((X + B)^2 - A - C), X3 = E^2 - 2D).
template <int H>
__device__ __noinline__ LinePart prep_dbl(Tw& t, Lane g) {
    level<H>(pick(g.k, t.x, t.y, t.z, t.y, t.x, t.x), pick(g.k, t.x, t.y, t.z, t.z, t.x, t.x), g);
    const Fq a = level_get(g, 0), b = level_get(g, 1), zz = level_get(g, 2);
    const Fq e = Fq::add(Fq::dbl(a), a), z3 = Fq::dbl(level_get(g, 3)), xb = Fq::add(t.x, b);
    level<H>(pick(g.k, b, xb, e, z3, e, e), pick(g.k, b, xb, zz, zz, t.x, e), g);
    const Fq c = level_get(g, 0), ezz = level_get(g, 2), z3zz = level_get(g, 3), ex = level_get(g, 4);
    const Fq d = Fq::dbl(Fq::sub(Fq::sub(level_get(g, 1), a), c));
    const Fq x3 = Fq::sub(level_get(g, 5), Fq::dbl(d));
    level<H>(e, Fq::sub(d, x3), g);
    t.y = Fq::sub(level_get(g, 0), Fq::dbl(Fq::dbl(Fq::dbl(c))));
    t.x = x3;
    t.z = z3;
    return {z3zz, Fq::neg(ezz), Fq::sub(ex, Fq::dbl(b))};
}
// T <- T + S (S affine) and its line, in five levels:
//   ZZ = Z^2; U2 = xs ZZ, ZZZ = Z ZZ;
//   S2 = ys ZZZ, HH = H^2, (Z + H)^2            (H = U2 - X);
//   J = H I, V = X I, r^2, r xs, Z3 ys          (I = 4 HH, r = 2(S2 - Y), Z3 = (Z + H)^2 - ZZ - HH);
//   r (V - X3), Y J                             (X3 = r^2 - J - 2V).
template <int H>
__device__ __noinline__ LinePart prep_add(Tw& t, Fq xs, Fq ys, Lane g) {
    level<H>(t.z, t.z, g);
    const Fq zz = level_get(g, 0);
    level<H>(pick(g.k, xs, t.z, xs, xs, xs, xs), zz, g);
    const Fq h = Fq::sub(level_get(g, 0), t.x), zh = Fq::add(t.z, h), zzz = level_get(g, 1);
    level<H>(pick(g.k, ys, h, zh, h, h, h), pick(g.k, zzz, h, zh, h, h, h), g);
    const Fq hh = level_get(g, 1);
    const Fq i = Fq::dbl(Fq::dbl(hh));
    const Fq r = Fq::dbl(Fq::sub(level_get(g, 0), t.y));
    const Fq z3 = Fq::sub(Fq::sub(level_get(g, 2), zz), hh);
    level<H>(pick(g.k, h, t.x, r, r, z3, r), pick(g.k, i, i, r, xs, ys, r), g);
    const Fq j = level_get(g, 0), vv = level_get(g, 1), rxs = level_get(g, 3), z3ys = level_get(g, 4);
    const Fq x3 = Fq::sub(Fq::sub(level_get(g, 2), j), Fq::dbl(vv));
    level<H>(pick(g.k, r, t.y, r, r, r, r), pick(g.k, Fq::sub(vv, x3), j, r, r, r, r), g);
    t.y = Fq::sub(level_get(g, 0), Fq::dbl(level_get(g, 1)));
    t.x = x3;
    t.z = z3;
    return {z3, Fq::neg(r), Fq::sub(rxs, z3ys)};
}
// The loop over the lines of Q in order: put(line) for each.
template <int H, class Put>
DV_INL void for_lines(const G2A& q, const Lane& g, Put&& put) {
    const Fq qx = g.c ? q.x.c1 : q.x.c0, qy = g.c ? q.y.c1 : q.y.c0, nqy = Fq::neg(qy);
    Tw t{qx, qy, g.c ? Fq::zero() : Fq::one()};
#pragma unroll 1
    for (int i = 1; i < NAF_LEN; ++i) {
        put(prep_dbl<H>(t, g), i > 1);
        const int d = NAF_6Z2[i];
        if (d) put(prep_add<H>(t, qx, d > 0 ? qy : nqy, g), false);
    }
    // pi(Q) = (conj(x) xi^((q-1)/3), conj(y) xi^((q-1)/2)); -pi^2(Q) = (x xi^((q^2-1)/3), -y xi^((q^2-1)/2))
    const Fq2 x1 = Fq2::mul(Fq2::conj(q.x), frob1(2)), y1 = Fq2::mul(Fq2::conj(q.y), frob1(3));
    put(prep_add<H>(t, g.c ? x1.c1 : x1.c0, g.c ? y1.c1 : y1.c0, g), false);
    put(prep_add<H>(t, Fq::mul(qx, frob2(2)), Fq::neg(Fq::mul(qy, frob2(3))), g), false);
}

// The LINES triples of every Q (one lane group each) at lines[LINES q ..],
// and inf[q] = 1 for Q at infinity (whose lines count as 1).
template <int H>
__global__ void __launch_bounds__(THREADS) k_prepare(const G2A* __restrict__ g2, uint64_t nq, Line* __restrict__ lines,
                                                     uint32_t* __restrict__ inf) {
    const Lane g = lane_setup<H>();
    const bool mine = g.writes && g.group < nq;
    const uint64_t qi = g.group < nq ? g.group : 0;
    const G2A q = g2[qi];
    if (mine && g.k == 0 && g.c == 0) inf[qi] = q.is_inf() ? 1u : 0u;
    Fq* out = reinterpret_cast<Fq*>(lines + (uint64_t)LINES * qi) + 2 * g.k + g.c;
    for_lines<H>(q, g, [&](const LinePart& l, bool) {
        if (mine && g.k < 3) *out = g.k == 0 ? l.a : g.k == 1 ? l.b : l.c;
        out += sizeof(Line) / sizeof(Fq);
    });
}

// This lane's component of a line scaled to P (on lanes k = 0, 1, 3): raw is
// its component of A, B or C; one: the line counts as 1.
DV_INL Fq scaled_line(const Lane& g, const Fq& raw, const Fq& coord, bool one) {
    const Fq s = Fq::mul(raw, coord);
    const Fq v = g.k == 3 ? raw : s;
    return one ? g_one(g) : v;
}

// Miller value of every equation from its terms' P and prepared Q, one lane
// group per equation and one f for all its terms (the multi-Miller loop):
// every step squares f once and multiplies in the lines of all the terms.
// Every group of a warp runs the warp's largest term count.  The next line
// and coordinate are loaded before the current product.  Component c of
// coefficient k of equation e at out[12 e + 2 k + c]; without offsets every
// term is its own equation (a group per term, for batches too small to fill
// the GPU, whose terms then meet in the final exponentiation).
// Measured (the terms of one proof's 49 equations): 909 us with six lanes a
// group and Karatsuba products, 343 us with H = 2.
template <int H>
__global__ void __launch_bounds__(THREADS) k_miller_multi(const G1A* __restrict__ g1,
                                                          const uint32_t* __restrict__ qidx,
                                                          const uint32_t* __restrict__ qinf,
                                                          const Line* __restrict__ lines,
                                                          const uint64_t* __restrict__ offsets, uint64_t equations,
                                                          Fq* __restrict__ out) {
    const Lane g = lane_setup<H>();
    const bool mine = g.group < equations;
    const uint64_t e = mine ? g.group : 0;
    const uint64_t first = !mine ? 0 : offsets ? offsets[e] : e;
    const uint64_t count = !mine ? 0 : offsets ? offsets[e + 1] - first : 1;
    uint64_t most = count;
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) {
        const uint64_t o = __shfl_xor_sync(FULL, most, off);
        most = o > most ? o : most;
    }
    // term j of this group at line n (term 0 of the call stands in past the
    // group's count, which is then nonzero somewhere in the warp)
    const int part = 2 * (g.k == 1 ? 1 : g.k == 3 ? 2 : 0) + g.c;
    auto fetch = [&](uint64_t j, int n, Fq& raw, Fq& coord, bool& one) {
        const bool have = j < count;
        const uint64_t t = have ? first + j : 0;
        const G1A p = g1[t];
        const uint32_t qi = qidx[t];
        raw = reinterpret_cast<const Fq*>(lines + (uint64_t)LINES * qi + n)[part];
        coord = g.k == 1 ? p.x : p.y;
        one = !have || p.is_inf() || qinf[qi] != 0;
    };
    Fq f = g_one(g);
    if (most) {
        Fq raw, coord;
        bool one;
        fetch(0, 0, raw, coord, one);
        int n = 0, extra = 0;  // extra: the step's second line (an addition) comes next
#pragma unroll 1
        for (int i = 1; n < LINES;) {
            if (i > 1 && i < NAF_LEN && !extra) f = g_sqr<H>(g, f);
#pragma unroll 1
            for (uint64_t j = 0; j < most; ++j) {
                const Fq r = raw, c = coord;
                const bool o = one;
                const bool last = j + 1 == most;
                if (!last || n + 1 < LINES) fetch(last ? 0 : j + 1, last ? n + 1 : n, raw, coord, one);
                f = g_mul_line<H>(g, f, scaled_line(g, r, c, o));
            }
            ++n;
            if (i < NAF_LEN && !extra && NAF_6Z2[i]) {
                extra = 1;
            } else {
                extra = 0;
                ++i;
            }
        }
    }
    if (mine && g.writes) out[12 * e + 2 * g.k + g.c] = f;
}

template <int H>
__device__ Fq g_final_exponentiation(Fq m, const Lane& g) {
    const auto mul = [&](const Fq& a, const Fq& b) { return g_mul<H>(g, a, b); };
    const auto sqr = [&](const Fq& a) { return g_cyc_sqr<H>(a, g); };
    Fq f = mul(g_conj(m, g.k), g_inv<H>(m, g));  // ^(q^6 - 1)
    f = mul(g_frob(g, f, 2), f);                  // ^(q^2 + 1)
    const Fq a = g_pow_z<H>(f, g);
    const Fq b = g_pow_z<H>(a, g);
    const Fq c = g_pow_z<H>(b, g);
    const Fq a2 = sqr(a), a4 = sqr(a2), a6 = mul(a4, a2);
    const Fq b2 = sqr(b), b6 = mul(sqr(b2), b2);
    const Fq b12 = sqr(b6);
    const Fq c4 = sqr(sqr(c)), c12 = mul(sqr(c4), c4);
    const Fq tt = mul(c12, b6);
    const Fq l1 = mul(tt, a4);
    const Fq l2 = mul(tt, a6);
    const Fq l3 = mul(l1, g_conj(f, g.k));
    const Fq l0 = mul(mul(mul(c12, b12), a6), f);
    Fq r = mul(l0, g_frob(g, l1, 1));
    r = mul(r, g_frob(g, l2, 2));
    return mul(r, g_frob(g, l3, 3));
}

// Miller value of every term, one lane group per term (layout as above),
// for G2 points that do not repeat; infinity on either side gives one.
template <int H>
__global__ void __launch_bounds__(THREADS) k_miller(const G1A* __restrict__ g1, const G2A* __restrict__ g2,
                                                    uint64_t terms, Fq* __restrict__ out) {
    const Lane g = lane_setup<H>();
    const bool mine = g.group < terms;
    const uint64_t t = mine ? g.group : 0;  // idle groups compute on term 0
    const G1A p = g1[t];
    const G2A q = g2[t];
    const Fq coord = g.k == 1 ? p.x : p.y;
    Fq f = g_one(g);
    for_lines<H>(q, g, [&](const LinePart& l, bool square) {
        if (square) f = g_sqr<H>(g, f);
        f = g_mul_line<H>(g, f, scaled_line(g, g.k == 0 ? l.a : g.k == 1 ? l.b : l.c, coord, false));
    });
    if (mine && g.writes) out[12 * t + 2 * g.k + g.c] = (p.is_inf() || q.is_inf()) ? g_one(g) : f;
}

// One lane group per equation: product of its terms' values (every group of
// a warp runs the warp's largest term count, multiplying by one past its
// own; without offsets one value per equation), final exponentiation,
// verdict, and with gt the canonical GT element.
// Measured (49 equations): 1383 us with six lanes a group, 488 us with H = 2.
template <int H>
__global__ void __launch_bounds__(THREADS) k_final_exp(const Fq* __restrict__ miller,
                                                       const uint64_t* __restrict__ offsets, uint64_t equations,
                                                       uint8_t* __restrict__ verdicts, uint8_t* __restrict__ gt) {
    const Lane g = lane_setup<H>();
    const bool mine = g.group < equations;
    const uint64_t e = mine ? g.group : 0;
    const uint64_t first = !mine ? 0 : offsets ? offsets[e] : e;
    const uint64_t count = !mine ? 0 : offsets ? offsets[e + 1] - first : 1;
    uint64_t most = count;
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) {
        const uint64_t o = __shfl_xor_sync(FULL, most, off);
        most = o > most ? o : most;
    }
    Fq f = g_one(g);
#pragma unroll 1
    for (uint64_t t = 0; t < most; ++t) {
        const Fq v = t < count ? miller[12 * (first + t) + 2 * g.k + g.c] : g_one(g);
        f = t == 0 ? v : g_mul<H>(g, f, v);
    }
    const Fq r = g_final_exponentiation<H>(f, g);
    const bool ok = g.k == 0 && g.c == 0 ? r == Fq::one() : r.is_zero();
    const unsigned all = __ballot_sync(FULL, ok) >> (H == 1 ? threadIdx.x & 16 : 0);
    if (!mine || !g.writes) return;
    if (verdicts && g.k == 0 && g.c == 0) verdicts[e] = (all & 0xfffu) == 0xfffu ? 1 : 0;
    if (gt) {
        // tower order: w^0, w^2, w^4, w^1, w^3, w^5
        const int slot = (g.k & 1) ? 3 + (g.k >> 1) : (g.k >> 1);
        store_canonical(gt + 384 * e + 64 * slot + 32 * g.c, r);
    }
}

constexpr uint64_t PREP_MAX = 1ull << 17;  // distinct G2 points prepared in one call (17.5 KB each)

// Whether a call of this many groups gives each the whole warp: while that
// leaves at most two warps on each SM quarter, where the multiply pipe is
// busy.  Limits of one, two and four warps measured the same to 1 % on one
// proof's checks and on 32 proofs'; 4096 equations take 3.78 ms (5.26 ms
// with six lanes a group), one alone 0.83 ms (2.82 ms).
constexpr uint64_t SPLIT_WARPS = 2;
bool split_groups(uint64_t groups) { return groups <= SPLIT_WARPS * 4 * (uint64_t)sm_count(); }
template <int H>
unsigned group_blocks(uint64_t groups) {
    return (unsigned)((groups + GROUPS_PER_BLOCK<H> - 1) / GROUPS_PER_BLOCK<H>);
}
void launch_prepare(const G2A* q, uint64_t nq, Line* lines, uint32_t* inf, cudaStream_t st) {
    if (split_groups(nq)) k_prepare<2><<<group_blocks<2>(nq), THREADS, SM_BYTES<2>, st>>>(q, nq, lines, inf);
    else k_prepare<1><<<group_blocks<1>(nq), THREADS, SM_BYTES<1>, st>>>(q, nq, lines, inf);
    DV_LAUNCH();
}
void launch_miller(const G1A* p, const G2A* q, uint64_t terms, Fq* out, cudaStream_t st) {
    if (split_groups(terms)) k_miller<2><<<group_blocks<2>(terms), THREADS, SM_BYTES<2>, st>>>(p, q, terms, out);
    else k_miller<1><<<group_blocks<1>(terms), THREADS, SM_BYTES<1>, st>>>(p, q, terms, out);
    DV_LAUNCH();
}
// d_off null: one group per term
void launch_miller_multi(const G1A* p, const uint32_t* qidx, const uint32_t* qinf, const Line* lines,
                         const uint64_t* d_off, uint64_t groups, Fq* out, cudaStream_t st) {
    if (split_groups(groups))
        k_miller_multi<2><<<group_blocks<2>(groups), THREADS, SM_BYTES<2>, st>>>(p, qidx, qinf, lines, d_off, groups, out);
    else
        k_miller_multi<1><<<group_blocks<1>(groups), THREADS, SM_BYTES<1>, st>>>(p, qidx, qinf, lines, d_off, groups, out);
    DV_LAUNCH();
}
void launch_final_exp(const Fq* mil, const uint64_t* d_off, uint64_t equations, uint8_t* verdicts, uint8_t* gt,
                      cudaStream_t st) {
    if (split_groups(equations))
        k_final_exp<2><<<group_blocks<2>(equations), THREADS, SM_BYTES<2>, st>>>(mil, d_off, equations, verdicts, gt);
    else
        k_final_exp<1><<<group_blocks<1>(equations), THREADS, SM_BYTES<1>, st>>>(mil, d_off, equations, verdicts, gt);
    DV_LAUNCH();
}

// Whether the prepared Miller loops run one group per equation (the
// multi-Miller loop, one square of f for all terms) rather than one per term
// (shorter chains): per equation once a group per term would take more than
// one wave of resident blocks.
bool miller_per_equation(uint64_t terms) {
    static const uint64_t wave = [] {
        int blocks = 0;
        DV_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k_miller_multi<1>, THREADS, SM_BYTES<1>));
        return (uint64_t)sm_count() * (uint64_t)std::max(1, blocks) * GROUPS_PER_BLOCK<1>;
    }();
    return terms > wave;
}

// 128-byte G2 wire points as hash keys (FNV-1a over the words).
struct G2Key {
    uint64_t w[16];
    bool operator==(const G2Key& o) const { return memcmp(w, o.w, sizeof(w)) == 0; }
};
struct G2KeyHash {
    size_t operator()(const G2Key& k) const {
        uint64_t h = 1469598103934665603ull;
        for (uint64_t x : k.w) h = (h ^ x) * 1099511628211ull;
        return (size_t)h;
    }
};

// Device copy of the equations' term offsets.
uint64_t* upload_offsets(Backend& b, const uint64_t* offsets, uint64_t equations, cudaStream_t st) {
    uint64_t* d_off = b.idx.as<uint64_t>(equations + 1);
    DV_CUDA(cudaMemcpyAsync(d_off, offsets, 8 * (equations + 1), cudaMemcpyHostToDevice, st));
    return d_off;
}

// Final exponentiation of the Miller values in mil (one per term, folded per
// equation by the device offsets d_off; one per equation when d_off is
// null), verdicts / GT elements back to the host.
void finish_equations(Backend& b, const Fq* mil, const uint64_t* d_off, uint64_t equations, uint8_t* verdicts,
                      uint8_t* gt, const uint32_t* bad, const std::vector<uint64_t>* g2_first, cudaStream_t st) {
    // GT elements first (16-byte aligned stores), then the verdict bytes
    uint8_t* d_gt = b.out_buf.as<uint8_t>(equations * ((gt ? 384 : 0) + 1));
    uint8_t* d_out = d_gt + (gt ? 384 * equations : 0);
    launch_final_exp(mil, d_off, equations, d_out, gt ? d_gt : nullptr, st);
    uint32_t hbad[2];
    DV_CUDA(cudaMemcpyAsync(hbad, bad, sizeof(hbad), cudaMemcpyDeviceToHost, st));
    DV_CUDA(cudaStreamSynchronize(st));
    if (hbad[0] != 0xffffffffu) throw InvalidArgument("invalid G1 point at term " + std::to_string(hbad[0]));
    if (hbad[1] != 0xffffffffu)
        throw InvalidArgument("invalid G2 point at term " +
                              std::to_string(g2_first ? (*g2_first)[hbad[1]] : (uint64_t)hbad[1]));
    if (verdicts) DV_CUDA(cudaMemcpy(verdicts, d_out, equations, cudaMemcpyDeviceToHost));
    if (gt) DV_CUDA(cudaMemcpy(gt, d_gt, 384 * equations, cudaMemcpyDeviceToHost));
}

}  // namespace

struct PreparedG2 {
    uint64_t n = 0;
    DevBuf points;  // G2A (Montgomery affine)
    DevBuf lines;   // LINES per point
    DevBuf inf;     // u32 per point: 1 at infinity
};
struct PairingState {
    std::map<uint64_t, std::unique_ptr<PreparedG2>> prepared;
    DevBuf lines, inf, qidx;
};

namespace {

PairingState& pairing_state(Backend& b) {
    if (!b.pairing) b.pairing = std::make_shared<PairingState>();
    return *b.pairing;
}

void pairing_run(Backend& b, const uint8_t* g1, const uint8_t* g2, uint64_t terms, const uint64_t* offsets,
                 uint64_t equations, uint8_t* verdicts, uint8_t* gt, cudaStream_t st) {
    // the distinct G2 points of the call: shared ones are prepared once
    std::vector<uint32_t> qidx;
    std::vector<uint64_t> first;
    std::vector<uint8_t> distinct;
    if (terms > 1) {
        std::unordered_map<G2Key, uint32_t, G2KeyHash> seen;
        seen.reserve(terms);
        qidx.resize(terms);
        for (uint64_t t = 0; t < terms; ++t) {
            G2Key key;
            memcpy(key.w, g2 + 128 * t, 128);
            const auto it = seen.emplace(key, (uint32_t)first.size());
            if (it.second) {
                first.push_back(t);
                distinct.insert(distinct.end(), g2 + 128 * t, g2 + 128 * (t + 1));
            }
            qidx[t] = it.first->second;
        }
    }
    const uint64_t nq = first.size();
    const bool prepared = terms > 1 && nq < terms && nq <= PREP_MAX;
    const bool multi = prepared && miller_per_equation(terms);
    const uint64_t g2_count = prepared ? nq : terms;
    uint8_t* d_in = b.in_points.as<uint8_t>(64 * terms + 128 * g2_count);
    DV_CUDA(cudaMemcpyAsync(d_in, g1, 64 * terms, cudaMemcpyHostToDevice, st));
    DV_CUDA(cudaMemcpyAsync(d_in + 64 * terms, prepared ? distinct.data() : g2, 128 * g2_count,
                            cudaMemcpyHostToDevice, st));
    G1A* p = b.conv_points.as<G1A>(terms + 2 * g2_count);  // G1A (64 B) then G2A (128 B)
    G2A* q = reinterpret_cast<G2A*>(p + terms);
    uint32_t* bad = b.err.as<uint32_t>(2);
    DV_CUDA(cudaMemsetAsync(bad, 0xff, 2 * sizeof(uint32_t), st));
    convert_points<Fq>(d_in, p, terms, bad, st);
    convert_points<Fq2>(d_in + 64 * terms, q, g2_count, bad + 1, st);
    uint64_t* d_off = upload_offsets(b, offsets, equations, st);
    Fq* mil = b.aux.as<Fq>(12 * std::max<uint64_t>(1, std::max(terms, equations)));
    if (prepared) {
        PairingState& ps = pairing_state(b);
        Line* lines = ps.lines.as<Line>((uint64_t)LINES * nq);
        uint32_t* qinf = ps.inf.as<uint32_t>(nq);
        uint32_t* d_qidx = ps.qidx.as<uint32_t>(terms);
        DV_CUDA(cudaMemcpyAsync(d_qidx, qidx.data(), 4 * terms, cudaMemcpyHostToDevice, st));
        launch_prepare(q, nq, lines, qinf, st);
        launch_miller_multi(p, d_qidx, qinf, lines, multi ? d_off : nullptr, multi ? equations : terms, mil, st);
    } else if (terms) {
        launch_miller(p, q, terms, mil, st);
    }
    finish_equations(b, mil, prepared && multi ? nullptr : d_off, equations, verdicts, gt, bad,
                     prepared ? &first : nullptr, st);
}

}  // namespace

// Bytes of one prepared G2 point (its Miller loop's line triples).
uint64_t pairing_prepared_bytes() { return (uint64_t)LINES * sizeof(Line); }

// Prepares nq Montgomery affine G2 points of q: their lines into `lines`
// (nq * pairing_prepared_bytes()) and a u32 per point into qinf (1 at
// infinity).  No host synchronisation; the buffers are the caller's, so a
// set of fixed points (a verifying key) can be prepared once and reused.
void pairing_prepare_device(const G2A* q, uint64_t nq, void* lines, uint32_t* qinf, cudaStream_t st) {
    if (!nq) return;
    if (nq > PREP_MAX) throw InvalidArgument("too many distinct G2 points in one check");
    launch_prepare(q, nq, static_cast<Line*>(lines), qinf, st);
}

// Pairing-product checks over prepared G2 points, with no host
// synchronisation: equation e holds iff prod over terms
// [d_off[e], d_off[e+1]) of e(p[k], Q[d_qidx[k]]) is one, where Q's lines
// and infinity flags are at lines / qinf (pairing_prepare_device);
// d_verdicts[e] = 1 / 0.  p: Montgomery affine G1 terms.  Scratch comes
// from the backend.
void pairing_check_prepared(Backend& b, const G1A* p, uint64_t terms, const void* lines, const uint32_t* qinf,
                            const uint32_t* d_qidx, const uint64_t* d_off, uint64_t equations, uint8_t* d_verdicts,
                            cudaStream_t st) {
    if (!equations) return;
    const Line* ln = static_cast<const Line*>(lines);
    Fq* mil = b.aux.as<Fq>(12 * std::max<uint64_t>(1, std::max(terms, equations)));
    const bool multi = miller_per_equation(terms);
    if (multi) launch_miller_multi(p, d_qidx, qinf, ln, d_off, equations, mil, st);
    else if (terms) launch_miller_multi(p, d_qidx, qinf, ln, nullptr, terms, mil, st);
    launch_final_exp(mil, multi ? nullptr : d_off, equations, d_verdicts, nullptr, st);
}

// The same checks with the nq G2 points of q prepared first (into the
// backend's pairing scratch).  For callers that build their equations on
// the device (the Dynaverse verifier, dynaverse.cu).
void pairing_check_device(Backend& b, const G1A* p, uint64_t terms, const G2A* q, uint64_t nq,
                          const uint32_t* d_qidx, const uint64_t* d_off, uint64_t equations, uint8_t* d_verdicts,
                          cudaStream_t st) {
    if (!equations) return;
    if (nq > PREP_MAX) throw InvalidArgument("too many distinct G2 points in one check");
    PairingState& ps = pairing_state(b);
    Line* lines = ps.lines.as<Line>((uint64_t)LINES * std::max<uint64_t>(1, nq));
    uint32_t* qinf = ps.inf.as<uint32_t>(std::max<uint64_t>(1, nq));
    pairing_prepare_device(q, nq, lines, qinf, st);
    pairing_check_prepared(b, p, terms, lines, qinf, d_qidx, d_off, equations, d_verdicts, st);
}

namespace {

void check_offsets(const uint64_t* offsets, size_t equations) {
    require(offsets && equations >= 1 && equations <= (1u << 24), "invalid pairing check arguments");
    require(offsets[0] == 0, "pairing offsets must start at 0");
    for (size_t e = 0; e < equations; ++e) require(offsets[e + 1] >= offsets[e], "pairing offsets must not decrease");
    require(offsets[equations] <= (1u << 24), "invalid pairing terms");
}

}  // namespace
}  // namespace dv

using namespace dv;

extern "C" int dvgpu_bn254_pairing_check(void* opaque, const uint8_t* g1, const uint8_t* g2, const uint64_t* offsets,
                                         size_t equations, uint8_t* verdicts, char* error, size_t cap) {
    return guarded(opaque, error, cap, [&](Backend& b) {
        check_offsets(offsets, equations);
        const uint64_t terms = offsets[equations];
        require(verdicts && (g1 || !terms) && (g2 || !terms), "invalid pairing terms");
        pairing_run(b, g1, g2, terms, offsets, equations, verdicts, nullptr, b.stream);
    });
}

extern "C" int dvgpu_bn254_pairing(void* opaque, const uint8_t* g1, const uint8_t* g2, size_t n, uint8_t* gt,
                                   char* error, size_t cap) {
    return guarded(opaque, error, cap, [&](Backend& b) {
        require(g1 && g2 && gt && n >= 1 && n <= (1u << 24), "invalid pairing arguments");
        std::vector<uint64_t> off(n + 1);
        for (size_t i = 0; i <= n; ++i) off[i] = i;
        pairing_run(b, g1, g2, n, off.data(), n, nullptr, gt, b.stream);
    });
}

extern "C" int dvgpu_bn254_g2_prepare(void* opaque, const uint8_t* g2, size_t n, uint64_t* prepared, char* error,
                                      size_t cap) {
    return guarded(opaque, error, cap, [&](Backend& b) {
        require(g2 && prepared && n >= 1 && n <= PREP_MAX, "invalid G2 preparation arguments (1..2^17 points)");
        const cudaStream_t st = b.stream;
        auto pg = std::make_unique<PreparedG2>();
        pg->n = n;
        uint8_t* d_in = b.in_points.as<uint8_t>(128 * n);
        DV_CUDA(cudaMemcpyAsync(d_in, g2, 128 * n, cudaMemcpyHostToDevice, st));
        uint32_t* bad = b.err.as<uint32_t>(1);
        DV_CUDA(cudaMemsetAsync(bad, 0xff, sizeof(uint32_t), st));
        G2A* q = pg->points.as<G2A>(n);
        convert_points<Fq2>(d_in, q, n, bad, st);
        launch_prepare(q, n, pg->lines.as<Line>((uint64_t)LINES * n), pg->inf.as<uint32_t>(n), st);
        const uint32_t first_bad = read_err_word(b, bad, st);
        if (first_bad != 0xffffffffu) throw InvalidArgument("invalid G2 point at index " + std::to_string(first_bad));
        const uint64_t h = b.next_handle++;
        pairing_state(b).prepared[h] = std::move(pg);
        *prepared = h;
    });
}

extern "C" int dvgpu_bn254_g2_prepared_release(void* opaque, uint64_t prepared, char* error, size_t cap) {
    return guarded(opaque, error, cap, [&](Backend& b) {
        PairingState& ps = pairing_state(b);
        require(ps.prepared.count(prepared) != 0, "unknown prepared G2 handle");
        DV_CUDA(cudaStreamSynchronize(b.stream));
        ps.prepared.erase(prepared);
    });
}

extern "C" int dvgpu_bn254_pairing_check_prepared(void* opaque, const uint8_t* g1, uint64_t prepared,
                                                  const uint32_t* q_index, const uint64_t* offsets, size_t equations,
                                                  uint8_t* verdicts, char* error, size_t cap) {
    return guarded(opaque, error, cap, [&](Backend& b) {
        check_offsets(offsets, equations);
        const uint64_t terms = offsets[equations];
        require(verdicts && ((g1 && q_index) || !terms), "invalid pairing terms");
        PairingState& ps = pairing_state(b);
        const auto it = ps.prepared.find(prepared);
        require(it != ps.prepared.end(), "unknown prepared G2 handle");
        const PreparedG2& pg = *it->second;
        for (uint64_t t = 0; t < terms; ++t) require(q_index[t] < pg.n, "prepared G2 index out of range");
        const cudaStream_t st = b.stream;
        uint8_t* d_in = b.in_points.as<uint8_t>(64 * terms);
        DV_CUDA(cudaMemcpyAsync(d_in, g1, 64 * terms, cudaMemcpyHostToDevice, st));
        G1A* p = b.conv_points.as<G1A>(std::max<uint64_t>(1, terms));
        uint32_t* bad = b.err.as<uint32_t>(2);
        DV_CUDA(cudaMemsetAsync(bad, 0xff, 2 * sizeof(uint32_t), st));
        convert_points<Fq>(d_in, p, terms, bad, st);
        uint64_t* d_off = upload_offsets(b, offsets, equations, st);
        Fq* mil = b.aux.as<Fq>(12 * std::max<uint64_t>(1, std::max(terms, equations)));
        uint32_t* d_qidx = ps.qidx.as<uint32_t>(std::max<uint64_t>(1, terms));
        if (terms) DV_CUDA(cudaMemcpyAsync(d_qidx, q_index, 4 * terms, cudaMemcpyHostToDevice, st));
        const bool multi = miller_per_equation(terms);
        // with no terms every equation's value is one (the kernels read only the offsets)
        if (terms)
            launch_miller_multi(p, d_qidx, pg.inf.view<uint32_t>(), pg.lines.view<Line>(), multi ? d_off : nullptr,
                                multi ? equations : terms, mil, st);
        finish_equations(b, mil, multi ? nullptr : d_off, equations, verdicts, nullptr, bad, nullptr, st);
    });
}
