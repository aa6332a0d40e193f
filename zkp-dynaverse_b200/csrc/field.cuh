// BN254 prime fields on sm_100a: 8 x 32-bit limbs, Montgomery form R = 2^256.
//
// Multiplication is CIOS (Koc, Acar, Kaliski, "Analyzing and comparing
// Montgomery multiplication algorithms", 1996) written as PTX carry chains.
// What bounds it is the 32x32 -> 64-bit multiply-add: four cycles a warp on
// each SM quarter with a carry or without, 6.2 for a lone warp; FP64
// products on 24-bit or 52-bit limbs come out no faster on this part, and
// share issue slots with the integer ones.  So the layout removes what is
// not a product:
//  - The running sum is two accumulators, T = E + 2^32 O, that take the
//    products with the even and with the odd limbs of a row.  A 64-bit product
//    then always lands on an even-aligned register pair (one multiply-add
//    instruction), also after the shift by one limb, which makes O the new
//    E and E without two limbs the new O: no moves, no re-split additions.
//    (Aligned and unaligned partial products in accumulators of their own:
//    Emmart, Luitjens, Weems and Woolley, "Optimizing modular multiplication for
//    NVIDIA's Maxwell GPUs", ARITH 2016, there for 16-bit halves.)
//  - With N = (p (-p^-1 mod 2^32) + 1) / 2^32, T + t0 p (-p^-1 mod 2^32) is
//    divisible by 2^32 and its quotient is (T >> 32) + t0 N (t0 the low limb):
//    a reduction step needs no product for its multiplier (Orup, "Simplifying
//    quotient determination in high-radix modular multiplication", ARITH
//    1995).  N < p, but the
//    steps no longer keep T below 2p, so the last two take the multiplier
//    m = -t0 / p mod 2^32 and p.  Bounds: T < 2^33 p < 2^288 before every
//    step, below 2p after the last.
// Measured (148 x 512 threads, pairs of products): 53.3 to 64.4 G products/s,
// against 68.8 that the multiply-adds alone would allow; one warp alone,
// 505 to 449 ns a product (single accumulator to this form).
//
// Values are kept fully reduced in [0, p).
#pragma once
#include <cstdint>

namespace dv {

struct FqCfg {
    static constexpr uint32_t P0 = 0xd87cfd47u, P1 = 0x3c208c16u, P2 = 0x6871ca8du, P3 = 0x97816a91u,
                              P4 = 0x8181585du, P5 = 0xb85045b6u, P6 = 0xe131a029u, P7 = 0x30644e72u;
    static constexpr uint32_t INV = 0xe4866389u;  // -p^{-1} mod 2^32
    static constexpr uint32_t ONE0 = 0xc58f0d9du, ONE1 = 0xd35d438du, ONE2 = 0xf5c70b3du, ONE3 = 0x0a78eb28u, ONE4 = 0x7879462cu, ONE5 = 0x666ea36fu, ONE6 = 0x9a07df2fu, ONE7 = 0x0e0a77c1u;
    static constexpr uint32_t R20 = 0x538afa89u, R21 = 0xf32cfc5bu, R22 = 0xd44501fbu, R23 = 0xb5e71911u, R24 = 0x0a417ff6u, R25 = 0x47ab1effu, R26 = 0xcab8351fu, R27 = 0x06d89f71u;
    static constexpr uint32_t R30 = 0xda1530dfu, R31 = 0xb1cd6dafu, R32 = 0xa7283db6u, R33 = 0x62f210e6u, R34 = 0x0ada0afbu, R35 = 0xef7f0b0cu, R36 = 0x2d592544u, R37 = 0x20fd6e90u;
};
struct FrCfg {
    static constexpr uint32_t P0 = 0xf0000001u, P1 = 0x43e1f593u, P2 = 0x79b97091u, P3 = 0x2833e848u,
                              P4 = 0x8181585du, P5 = 0xb85045b6u, P6 = 0xe131a029u, P7 = 0x30644e72u;
    static constexpr uint32_t INV = 0xefffffffu;
    static constexpr uint32_t ONE0 = 0x4ffffffbu, ONE1 = 0xac96341cu, ONE2 = 0x9f60cd29u, ONE3 = 0x36fc7695u, ONE4 = 0x7879462eu, ONE5 = 0x666ea36fu, ONE6 = 0x9a07df2fu, ONE7 = 0x0e0a77c1u;
    static constexpr uint32_t R20 = 0xae216da7u, R21 = 0x1bb8e645u, R22 = 0xe35c59e3u, R23 = 0x53fe3ab1u, R24 = 0x53bb8085u, R25 = 0x8c49833du, R26 = 0x7f4e44a5u, R27 = 0x0216d0b1u;
    static constexpr uint32_t R30 = 0xb4bf0040u, R31 = 0x5e94d8e1u, R32 = 0x1cfbb6b8u, R33 = 0x2a489cbeu, R34 = 0xa19fcfedu, R35 = 0x893cc664u, R36 = 0x7fcc657cu, R37 = 0x0cf8594bu;
};

#define DV_INL __device__ __forceinline__

// Operands of a 16-word asm statement r <- a op b.
#define DV_WIDE_OPERANDS(r, a, b)                                                                                     \
    : "=&r"(r.v[0]), "=&r"(r.v[1]), "=&r"(r.v[2]), "=&r"(r.v[3]), "=&r"(r.v[4]), "=&r"(r.v[5]), "=&r"(r.v[6]),       \
      "=&r"(r.v[7]), "=&r"(r.v[8]), "=&r"(r.v[9]), "=&r"(r.v[10]), "=&r"(r.v[11]), "=&r"(r.v[12]), "=&r"(r.v[13]),   \
      "=&r"(r.v[14]), "=&r"(r.v[15])                                                                                  \
    : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]), "r"(a.v[7]),        \
      "r"(a.v[8]), "r"(a.v[9]), "r"(a.v[10]), "r"(a.v[11]), "r"(a.v[12]), "r"(a.v[13]), "r"(a.v[14]), "r"(a.v[15]),  \
      "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]), "r"(b.v[4]), "r"(b.v[5]), "r"(b.v[6]), "r"(b.v[7]),        \
      "r"(b.v[8]), "r"(b.v[9]), "r"(b.v[10]), "r"(b.v[11]), "r"(b.v[12]), "r"(b.v[13]), "r"(b.v[14]), "r"(b.v[15])

// Two results of a paired multiplication.
template <class T>
struct PairOf {
    T r0, r1;
};

template <class C>
struct __align__(16) Fp {  // 16-byte aligned: global copies move as 128-bit accesses
    uint32_t v[8];

    DV_INL static Fp zero() {
        Fp r;
#pragma unroll
        for (int i = 0; i < 8; ++i) r.v[i] = 0;
        return r;
    }
    DV_INL static Fp one() {
        Fp r;
        r.v[0] = C::ONE0; r.v[1] = C::ONE1; r.v[2] = C::ONE2; r.v[3] = C::ONE3;
        r.v[4] = C::ONE4; r.v[5] = C::ONE5; r.v[6] = C::ONE6; r.v[7] = C::ONE7;
        return r;
    }
    // R^2 mod p: the Montgomery form of R.
    DV_INL static Fp r2() {
        Fp r;
        r.v[0] = C::R20; r.v[1] = C::R21; r.v[2] = C::R22; r.v[3] = C::R23;
        r.v[4] = C::R24; r.v[5] = C::R25; r.v[6] = C::R26; r.v[7] = C::R27;
        return r;
    }
    DV_INL bool is_zero() const {
        uint32_t x = v[0] | v[1] | v[2] | v[3] | v[4] | v[5] | v[6] | v[7];
        return x == 0;
    }
    DV_INL bool operator==(const Fp& o) const {
        uint32_t x = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) x |= v[i] ^ o.v[i];
        return x == 0;
    }

    // r = a - p if a >= p else a   (a < 2^256)
    DV_INL static void reduce_once(uint32_t* t) {
        uint32_t s[8], borrow;
        asm("sub.cc.u32 %0, %9, %17;\n\t"
            "subc.cc.u32 %1, %10, %18;\n\t"
            "subc.cc.u32 %2, %11, %19;\n\t"
            "subc.cc.u32 %3, %12, %20;\n\t"
            "subc.cc.u32 %4, %13, %21;\n\t"
            "subc.cc.u32 %5, %14, %22;\n\t"
            "subc.cc.u32 %6, %15, %23;\n\t"
            "subc.cc.u32 %7, %16, %24;\n\t"
            "subc.u32 %8, 0, 0;"
            : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6]),
              "=r"(s[7]), "=r"(borrow)
            : "r"(t[0]), "r"(t[1]), "r"(t[2]), "r"(t[3]), "r"(t[4]), "r"(t[5]), "r"(t[6]), "r"(t[7]),
              "n"(C::P0), "n"(C::P1), "n"(C::P2), "n"(C::P3), "n"(C::P4), "n"(C::P5), "n"(C::P6),
              "n"(C::P7));
        // borrow == 0xffffffff  <=>  t < p  -> keep t
#pragma unroll
        for (int i = 0; i < 8; ++i) t[i] = borrow ? t[i] : s[i];
    }

    DV_INL static Fp add(const Fp& a, const Fp& b) {
        Fp r = add_raw(a, b);
        reduce_once(r.v);
        return r;
    }

    DV_INL static Fp sub(const Fp& a, const Fp& b) {
        Fp r;
        uint32_t borrow;
        asm("sub.cc.u32 %0, %9, %17;\n\t"
            "subc.cc.u32 %1, %10, %18;\n\t"
            "subc.cc.u32 %2, %11, %19;\n\t"
            "subc.cc.u32 %3, %12, %20;\n\t"
            "subc.cc.u32 %4, %13, %21;\n\t"
            "subc.cc.u32 %5, %14, %22;\n\t"
            "subc.cc.u32 %6, %15, %23;\n\t"
            "subc.cc.u32 %7, %16, %24;\n\t"
            "subc.u32 %8, 0, 0;"
            : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]),
              "=r"(r.v[6]), "=r"(r.v[7]), "=r"(borrow)
            : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]),
              "r"(a.v[7]), "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]), "r"(b.v[4]), "r"(b.v[5]),
              "r"(b.v[6]), "r"(b.v[7]));
        // add back p & borrow
        asm("add.cc.u32 %0, %0, %8;\n\t"
            "addc.cc.u32 %1, %1, %9;\n\t"
            "addc.cc.u32 %2, %2, %10;\n\t"
            "addc.cc.u32 %3, %3, %11;\n\t"
            "addc.cc.u32 %4, %4, %12;\n\t"
            "addc.cc.u32 %5, %5, %13;\n\t"
            "addc.cc.u32 %6, %6, %14;\n\t"
            "addc.u32 %7, %7, %15;"
            : "+r"(r.v[0]), "+r"(r.v[1]), "+r"(r.v[2]), "+r"(r.v[3]), "+r"(r.v[4]), "+r"(r.v[5]),
              "+r"(r.v[6]), "+r"(r.v[7])
            : "r"(C::P0 & borrow), "r"(C::P1 & borrow), "r"(C::P2 & borrow), "r"(C::P3 & borrow),
              "r"(C::P4 & borrow), "r"(C::P5 & borrow), "r"(C::P6 & borrow), "r"(C::P7 & borrow));
        return r;
    }

    DV_INL static Fp dbl(const Fp& a) { return add(a, a); }

    DV_INL static Fp neg(const Fp& a) {
        Fp z = zero();
        return a.is_zero() ? a : sub(z, a);
    }

    // T = a b_0, then eight steps of reduction, the first seven each followed by T += a b_(i+1).
    DV_INL static Fp mul_inl(const Fp& a, const Fp& b) {
        Fp r = mul_lazy(a, b);
        reduce_once(r.v);
        return r;
    }
    // The same without the last subtraction.  The rows are a's, so the order
    // matters.  a < p and b < 4p: below 1.76 p, with T below 1.94 p 2^32.  a < 2p and
    // b < p: below 1.38 p, with T below 2.94 p 2^32 < 2^288.
    DV_INL static Fp mul_lazy(const Fp& a, const Fp& b) {
        constexpr Words N = reduction_words();
        uint32_t e[8], o[8], t[8];
        mul4(e, a.v[0], a.v[2], a.v[4], a.v[6], b.v[0]);
        mul4(o, a.v[1], a.v[3], a.v[5], a.v[7], b.v[0]);
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            const uint32_t t0 = e[0];
            shift_mac4(t, o, e, N.v[1], N.v[3], N.v[5], N.v[7], t0);
            mac4_top(o, t[7], N.v[0], N.v[2], N.v[4], N.v[6], t0);
            mac4(t, a.v[1], a.v[3], a.v[5], a.v[7], b.v[i + 1]);
            mac4_top(o, t[7], a.v[0], a.v[2], a.v[4], a.v[6], b.v[i + 1]);
            rotate(e, o, t);
        }
        reduce_step(e, o);
        shift_mac4(t, o, e, a.v[1], a.v[3], a.v[5], a.v[7], b.v[7]);
        mac4_top(o, t[7], a.v[0], a.v[2], a.v[4], a.v[6], b.v[7]);
        rotate(e, o, t);
        reduce_step(e, o);
        Fp r;
        merge(r.v, e, o);
        return r;
    }

    // One out-of-line copy of the multiplication keeps the point-arithmetic
    // loops inside the instruction cache (measured faster than inlining ten
    // ~300-instruction bodies per XYZZ addition).
#ifndef DV_MUL_INLINE
    __device__ __noinline__ static Fp mul(Fp a, Fp b) { return mul_inl(a, b); }
#else
    DV_INL static Fp mul(const Fp& a, const Fp& b) { return mul_inl(a, b); }
#endif
    // Two independent products in one out-of-line body: the compiler
    // interleaves their carry chains, which hides the multiply latency that a
    // lone chain exposes when few warps are resident.
    typedef PairOf<Fp> Pair;
#ifndef DV_MUL_INLINE
    __device__ __noinline__ static Pair mul2(Fp a, Fp b, Fp c, Fp d) { return {mul_inl(a, b), mul_inl(c, d)}; }
#else
    DV_INL static Pair mul2(const Fp& a, const Fp& b, const Fp& c, const Fp& d) {
        return {mul_inl(a, b), mul_inl(c, d)};
    }
#endif
    // 512-bit values: products that are added or subtracted before one
    // reduction (redc) instead of one each.
    struct Wide {
        uint32_t v[16];
    };
    DV_INL static Wide mul_wide(const Fp& a, const Fp& b) {
        const uint32_t ae[4] = {a.v[0], a.v[2], a.v[4], a.v[6]}, ao[4] = {a.v[1], a.v[3], a.v[5], a.v[7]};
        uint32_t e[17], o[17];  // word 16 only ever takes zero carries
#pragma unroll
        for (int j = 8; j < 17; ++j) e[j] = o[j] = 0;
        mul4(e, ae[0], ae[1], ae[2], ae[3], b.v[0]);
        mul4(o, ao[0], ao[1], ao[2], ao[3], b.v[0]);
#pragma unroll
        for (int i = 1; i < 8; ++i) {
            if (i & 1) {  // even limbs of a at odd positions, odd limbs at even ones
                chain<4>(o + i - 1, ae, b.v[i], o[i + 7]);
                chain<4>(e + i + 1, ao, b.v[i], e[i + 9 < 16 ? i + 9 : 16]);
            } else {
                chain<4>(e + i, ae, b.v[i], e[i + 8]);
                chain<4>(o + i, ao, b.v[i], o[i + 8]);
            }
        }
        return combine(e, o);
    }
    // a^2 as rows a_i (a_i, then the doubled limbs above i): 36 products.
    DV_INL static Wide sqr_wide(const Fp& a) {
        uint32_t e[17], o[17], d[8], s[8];  // d: limbs of 2a; s: a_j << 1, without the bit from below
#pragma unroll
        for (int j = 1; j < 8; ++j) {
            d[j] = __funnelshift_l(a.v[j - 1], a.v[j], 1);
            s[j] = a.v[j] << 1;
        }
#pragma unroll
        for (int j = 0; j < 17; ++j) e[j] = o[j] = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            uint32_t x[4] = {a.v[i], 0, 0, 0}, y[4] = {0, 0, 0, 0};
            int nx = 1, ny = 0;
            if (i < 7) y[ny++] = s[i + 1];
#pragma unroll
            for (int j = i + 2; j < 8; j += 2) x[nx++] = d[j];
#pragma unroll
            for (int j = i + 3; j < 8; j += 2) y[ny++] = d[j];
            if (nx == 4) chain<4>(e + 2 * i, x, a.v[i], e[2 * i + 8]);
            else if (nx == 3) chain<3>(e + 2 * i, x, a.v[i], e[2 * i + 6]);
            else if (nx == 2) chain<2>(e + 2 * i, x, a.v[i], e[2 * i + 4]);
            else chain<1>(e + 2 * i, x, a.v[i], e[2 * i + 2]);
            if (ny == 4) chain<4>(o + 2 * i, y, a.v[i], o[2 * i + 8]);
            else if (ny == 3) chain<3>(o + 2 * i, y, a.v[i], o[2 * i + 6]);
            else if (ny == 2) chain<2>(o + 2 * i, y, a.v[i], o[2 * i + 4]);
            else if (ny == 1) chain<1>(o + 2 * i, y, a.v[i], o[2 * i + 2]);
        }
        return combine(e, o);
    }
    // a + b and a - b modulo 2^512 (two's complement)
    DV_INL static Wide wide_add(const Wide& a, const Wide& b) {
        Wide r;
        asm("add.cc.u32 %0, %16, %32;\n\taddc.cc.u32 %1, %17, %33;\n\taddc.cc.u32 %2, %18, %34;\n\t"
            "addc.cc.u32 %3, %19, %35;\n\taddc.cc.u32 %4, %20, %36;\n\taddc.cc.u32 %5, %21, %37;\n\t"
            "addc.cc.u32 %6, %22, %38;\n\taddc.cc.u32 %7, %23, %39;\n\taddc.cc.u32 %8, %24, %40;\n\t"
            "addc.cc.u32 %9, %25, %41;\n\taddc.cc.u32 %10, %26, %42;\n\taddc.cc.u32 %11, %27, %43;\n\t"
            "addc.cc.u32 %12, %28, %44;\n\taddc.cc.u32 %13, %29, %45;\n\taddc.cc.u32 %14, %30, %46;\n\t"
            "addc.u32 %15, %31, %47;" DV_WIDE_OPERANDS(r, a, b));
        return r;
    }
    DV_INL static Wide wide_sub(const Wide& a, const Wide& b) {
        Wide r;
        asm("sub.cc.u32 %0, %16, %32;\n\tsubc.cc.u32 %1, %17, %33;\n\tsubc.cc.u32 %2, %18, %34;\n\t"
            "subc.cc.u32 %3, %19, %35;\n\tsubc.cc.u32 %4, %20, %36;\n\tsubc.cc.u32 %5, %21, %37;\n\t"
            "subc.cc.u32 %6, %22, %38;\n\tsubc.cc.u32 %7, %23, %39;\n\tsubc.cc.u32 %8, %24, %40;\n\t"
            "subc.cc.u32 %9, %25, %41;\n\tsubc.cc.u32 %10, %26, %42;\n\tsubc.cc.u32 %11, %27, %43;\n\t"
            "subc.cc.u32 %12, %28, %44;\n\tsubc.cc.u32 %13, %29, %45;\n\tsubc.cc.u32 %14, %30, %46;\n\t"
            "subc.u32 %15, %31, %47;" DV_WIDE_OPERANDS(r, a, b));
        return r;
    }
    // A negative t in (-2^255 p, 0) made non-negative by adding 2^255 p.
    // Differences of up to two products each way qualify: 2 p^2 < 2^255 p.
    DV_INL static void make_positive(Wide& t) {
        const uint32_t neg = (uint32_t)((int32_t)t.v[15] >> 31);
        const uint32_t p[8] = {C::P0, C::P1, C::P2, C::P3, C::P4, C::P5, C::P6, C::P7};
        uint32_t q[9];  // 2^31 p: words 7..15 of 2^255 p
        q[0] = (p[0] << 31) & neg;
#pragma unroll
        for (int j = 1; j < 8; ++j) q[j] = ((p[j] << 31) | (p[j - 1] >> 1)) & neg;
        q[8] = (p[7] >> 1) & neg;
        asm("add.cc.u32 %0, %0, %9;\n\taddc.cc.u32 %1, %1, %10;\n\taddc.cc.u32 %2, %2, %11;\n\t"
            "addc.cc.u32 %3, %3, %12;\n\taddc.cc.u32 %4, %4, %13;\n\taddc.cc.u32 %5, %5, %14;\n\t"
            "addc.cc.u32 %6, %6, %15;\n\taddc.cc.u32 %7, %7, %16;\n\taddc.u32 %8, %8, %17;"
            : "+r"(t.v[7]), "+r"(t.v[8]), "+r"(t.v[9]), "+r"(t.v[10]), "+r"(t.v[11]), "+r"(t.v[12]), "+r"(t.v[13]),
              "+r"(t.v[14]), "+r"(t.v[15])
            : "r"(q[0]), "r"(q[1]), "r"(q[2]), "r"(q[3]), "r"(q[4]), "r"(q[5]), "r"(q[6]), "r"(q[7]), "r"(q[8]));
    }
    // t / 2^256 mod p for 0 <= t < 2^255 p: the low half is reduced by itself
    // to at most p + p / 2^32, and with the high half (below p / 2) the sum
    // stays below 2p.
    DV_INL static Fp redc(const Wide& w) {
        Fp r = redc_raw(w);
        reduce_once(r.v);
        return r;
    }
    // The same without the last subtraction, for a high half of up to 4.27 p
    // (the sum then stays below 2^256 = 5.29 p).
    DV_INL static Fp redc_raw(const Wide& w) {
        constexpr Words N = reduction_words();
        uint32_t e[8], o[8], t[8];
        {
            const uint32_t t0 = w.v[0];
            asm("mad.lo.cc.u32 %0, %8, %12, %13;\n\tmadc.hi.u32 %1, %8, %12, 0;\n\t"
                "mul.lo.u32 %2, %9, %12;\n\tmul.hi.u32 %3, %9, %12;\n\t"
                "mul.lo.u32 %4, %10, %12;\n\tmul.hi.u32 %5, %10, %12;\n\t"
                "mul.lo.u32 %6, %11, %12;\n\tmul.hi.u32 %7, %11, %12;"
                : "=&r"(e[0]), "=&r"(e[1]), "=&r"(e[2]), "=&r"(e[3]), "=&r"(e[4]), "=&r"(e[5]), "=&r"(e[6]),
                  "=&r"(e[7])
                : "r"(N.v[0]), "r"(N.v[2]), "r"(N.v[4]), "r"(N.v[6]), "r"(t0), "r"(w.v[1]));
#pragma unroll
            for (int j = 0; j < 6; ++j) o[j] = w.v[j + 2];
            o[6] = o[7] = 0;
            mac4(o, N.v[1], N.v[3], N.v[5], N.v[7], t0);
        }
#pragma unroll
        for (int i = 1; i < 6; ++i) {
            const uint32_t t0 = e[0];
            shift_mac4(t, o, e, N.v[1], N.v[3], N.v[5], N.v[7], t0);
            mac4_top(o, t[7], N.v[0], N.v[2], N.v[4], N.v[6], t0);
            rotate(e, o, t);
        }
        reduce_step(e, o);
        const uint32_t m = (o[0] + e[1]) * C::INV;
        shift_mac4(t, o, e, C::P1, C::P3, C::P5, C::P7, m);
        mac4_top(o, t[7], C::P0, C::P2, C::P4, C::P6, m);
        rotate(e, o, t);
        uint32_t q[8];
        merge(q, e, o);
        Fp r;
        asm("add.cc.u32 %0, %8, %16;\n\taddc.cc.u32 %1, %9, %17;\n\taddc.cc.u32 %2, %10, %18;\n\t"
            "addc.cc.u32 %3, %11, %19;\n\taddc.cc.u32 %4, %12, %20;\n\taddc.cc.u32 %5, %13, %21;\n\t"
            "addc.cc.u32 %6, %14, %22;\n\taddc.u32 %7, %15, %23;"
            : "=&r"(r.v[0]), "=&r"(r.v[1]), "=&r"(r.v[2]), "=&r"(r.v[3]), "=&r"(r.v[4]), "=&r"(r.v[5]),
              "=&r"(r.v[6]), "=&r"(r.v[7])
            : "r"(q[0]), "r"(q[1]), "r"(q[2]), "r"(q[3]), "r"(q[4]), "r"(q[5]), "r"(q[6]), "r"(q[7]), "r"(w.v[8]),
              "r"(w.v[9]), "r"(w.v[10]), "r"(w.v[11]), "r"(w.v[12]), "r"(w.v[13]), "r"(w.v[14]), "r"(w.v[15]));
        return r;
    }
    // Montgomery square: 36 products and the reduction, against a product's 64.
    DV_INL static Fp sqr_inl(const Fp& a) { return redc(sqr_wide(a)); }
#ifndef DV_MUL_INLINE
    __device__ __noinline__ static Fp sqr(Fp a) { return sqr_inl(a); }
    // two independent squares in one body, like mul2
    __device__ __noinline__ static Pair sqr2(Fp a, Fp b) { return {sqr_inl(a), sqr_inl(b)}; }
#else
    DV_INL static Fp sqr(const Fp& a) { return sqr_inl(a); }
    DV_INL static Pair sqr2(const Fp& a, const Fp& b) { return {sqr_inl(a), sqr_inl(b)}; }
#endif

    // a b - c d with one reduction (200 multiply-adds against 272 for two
    // products): 1961 against 2355 ns for the pair at 148 x 512 threads.
    DV_INL static Fp mul_sub_inl(const Fp& a, const Fp& b, const Fp& c, const Fp& d) {
        Wide t = wide_sub(mul_wide(a, b), mul_wide(c, d));
        make_positive(t);
        return redc(t);
    }
#ifndef DV_MUL_INLINE
    __device__ __noinline__ static Fp mul_sub(Fp a, Fp b, Fp c, Fp d) { return mul_sub_inl(a, b, c, d); }
#else
    DV_INL static Fp mul_sub(const Fp& a, const Fp& b, const Fp& c, const Fp& d) { return mul_sub_inl(a, b, c, d); }
#endif
    // a + b without the reduction (a + b < 2^256), an operand of mul_wide
    DV_INL static Fp add_raw(const Fp& a, const Fp& b) {
        Fp r;
        asm("add.cc.u32 %0, %8, %16;\n\t"
            "addc.cc.u32 %1, %9, %17;\n\t"
            "addc.cc.u32 %2, %10, %18;\n\t"
            "addc.cc.u32 %3, %11, %19;\n\t"
            "addc.cc.u32 %4, %12, %20;\n\t"
            "addc.cc.u32 %5, %13, %21;\n\t"
            "addc.cc.u32 %6, %14, %22;\n\t"
            "addc.u32 %7, %15, %23;"
            : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]),
              "=r"(r.v[6]), "=r"(r.v[7])
            : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]),
              "r"(a.v[7]), "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]), "r"(b.v[4]), "r"(b.v[5]),
              "r"(b.v[6]), "r"(b.v[7]));
        return r;
    }

    // Values below 2p: a less 2p where it is not (a < 4p), and a - b + 2p < 4p.
    DV_INL static Fp reduce_2p(const Fp& a) {
        const Fp t = sub_raw(a, twice_modulus());
        const bool keep = (int32_t)t.v[7] < 0;  // a < 2p: the difference is negative, and 2p < 2^255
        Fp r;
#pragma unroll
        for (int i = 0; i < 8; ++i) r.v[i] = keep ? a.v[i] : t.v[i];
        return r;
    }
    DV_INL static Fp sub_2p(const Fp& a, const Fp& b) { return sub_raw(add_raw(a, twice_modulus()), b); }
    DV_INL static Fp twice_modulus() {
        const uint32_t p[8] = {C::P0, C::P1, C::P2, C::P3, C::P4, C::P5, C::P6, C::P7};
        Fp r;
        r.v[0] = p[0] << 1;
#pragma unroll
        for (int i = 1; i < 8; ++i) r.v[i] = (p[i] << 1) | (p[i - 1] >> 31);
        return r;
    }
    // a - b modulo 2^256
    DV_INL static Fp sub_raw(const Fp& a, const Fp& b) {
        Fp r;
        asm("sub.cc.u32 %0, %8, %16;\n\t"
            "subc.cc.u32 %1, %9, %17;\n\t"
            "subc.cc.u32 %2, %10, %18;\n\t"
            "subc.cc.u32 %3, %11, %19;\n\t"
            "subc.cc.u32 %4, %12, %20;\n\t"
            "subc.cc.u32 %5, %13, %21;\n\t"
            "subc.cc.u32 %6, %14, %22;\n\t"
            "subc.u32 %7, %15, %23;"
            : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]),
              "=r"(r.v[6]), "=r"(r.v[7])
            : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]),
              "r"(a.v[7]), "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]), "r"(b.v[4]), "r"(b.v[5]),
              "r"(b.v[6]), "r"(b.v[7]));
        return r;
    }
    DV_INL static Fp modulus() {
        Fp r;
        r.v[0] = C::P0; r.v[1] = C::P1; r.v[2] = C::P2; r.v[3] = C::P3;
        r.v[4] = C::P4; r.v[5] = C::P5; r.v[6] = C::P6; r.v[7] = C::P7;
        return r;
    }

    // Canonical little-endian limbs <-> Montgomery form.
    DV_INL static Fp from_canonical(const uint32_t* c) {
        Fp a;
#pragma unroll
        for (int i = 0; i < 8; ++i) a.v[i] = c[i];
        return mul(a, r2());
    }
    DV_INL void to_canonical(uint32_t* c) const {
        Fp one_raw = zero();
        one_raw.v[0] = 1;
        Fp r = mul(*this, one_raw);
#pragma unroll
        for (int i = 0; i < 8; ++i) c[i] = r.v[i];
    }
    // Canonical check: c < p.
    DV_INL static bool is_canonical(const uint32_t* c) {
        const uint32_t p[8] = {C::P0, C::P1, C::P2, C::P3, C::P4, C::P5, C::P6, C::P7};
#pragma unroll
        for (int i = 7; i >= 0; --i) {
            if (c[i] < p[i]) return true;
            if (c[i] > p[i]) return false;
        }
        return false;
    }

    // a^e for a 256-bit exponent given as 8 little-endian limbs.
    DV_INL static Fp pow(const Fp& a, const uint32_t* e) {
        Fp r = one();
        for (int i = 255; i >= 0; --i) {
            r = sqr(r);
            if ((e[i >> 5] >> (i & 31)) & 1) r = mul(r, a);
        }
        return r;
    }
    // 1 / a (0 for a = 0) by the divsteps of Bernstein and Yang ("Fast
    // constant-time gcd computation and modular inversion", TCHES 2019),
    // run variable-time: with f = p, g = aR, d = 0, e = 1 (f = d aR and
    // g = e aR mod p throughout), each batch takes 30 divsteps on the low 30
    // bits of f and g into a transition matrix scaled by 2^30, then applies
    // it to f, g (exact division by 2^30) and to d, e (division by 2^30 mod
    // p, adding md p with md = -(u d + v e) p^-1 mod 2^30).  Numbers are 9
    // limbs of 30 bits, the top one signed.  736 divsteps bring g to 0 for
    // inputs below 2^254, so 25 batches bound the loop, which ends when
    // g = 0.  Then f = +-1 and (aR)^-1 = f d with |d| < 26 p; the
    // Montgomery product with R^3 mod p turns (aR)^-1 into a^-1 R.
    DV_INL static Fp inv(const Fp& a) {
        constexpr uint32_t M30 = (1u << 30) - 1;
        constexpr uint32_t PINV30 = (0u - C::INV) & M30;  // p^-1 mod 2^30
        N9 f, g, d, e;
#pragma unroll
        for (int i = 0; i < 9; ++i) {
            f.l[i] = limb30(i);
            d.l[i] = 0;
            e.l[i] = i == 0;
            g.l[i] = (int32_t)(bits30(a, i));
        }
        int delta = 1;
#pragma unroll 1
        for (int batch = 0; batch < 25 && g.nonzero(); ++batch) {
            int32_t t[4];
            delta = divsteps30(delta, (uint32_t)f.l[0], (uint32_t)g.l[0], t);
            // (f, g) <- t (f, g) / 2^30 exactly; (d, e) <- t (d, e) / 2^30 mod p
            int64_t cf = (int64_t)t[0] * f.l[0] + (int64_t)t[1] * g.l[0];
            int64_t cg = (int64_t)t[2] * f.l[0] + (int64_t)t[3] * g.l[0];
            int64_t cd = (int64_t)t[0] * d.l[0] + (int64_t)t[1] * e.l[0];
            int64_t ce = (int64_t)t[2] * d.l[0] + (int64_t)t[3] * e.l[0];
            const int32_t md = (int32_t)((0u - (uint32_t)cd * PINV30) & M30);
            const int32_t me = (int32_t)((0u - (uint32_t)ce * PINV30) & M30);
            cd += (int64_t)md * limb30(0);
            ce += (int64_t)me * limb30(0);
            cf >>= 30;
            cg >>= 30;
            cd >>= 30;
            ce >>= 30;
#pragma unroll
            for (int i = 1; i < 9; ++i) {
                cf += (int64_t)t[0] * f.l[i] + (int64_t)t[1] * g.l[i];
                cg += (int64_t)t[2] * f.l[i] + (int64_t)t[3] * g.l[i];
                cd += (int64_t)t[0] * d.l[i] + (int64_t)t[1] * e.l[i] + (int64_t)md * limb30(i);
                ce += (int64_t)t[2] * d.l[i] + (int64_t)t[3] * e.l[i] + (int64_t)me * limb30(i);
                f.l[i - 1] = (int32_t)((uint32_t)cf & M30);
                g.l[i - 1] = (int32_t)((uint32_t)cg & M30);
                d.l[i - 1] = (int32_t)((uint32_t)cd & M30);
                e.l[i - 1] = (int32_t)((uint32_t)ce & M30);
                cf >>= 30;
                cg >>= 30;
                cd >>= 30;
                ce >>= 30;
            }
            f.l[8] = (int32_t)cf;
            g.l[8] = (int32_t)cg;
            d.l[8] = (int32_t)cd;
            e.l[8] = (int32_t)ce;
        }
        // x = 32 p + f d in (6 p, 58 p), then conditional subtractions of 32 p .. p
        const bool neg = f.l[8] < 0;
        N9 x;
        int64_t c = 0;
#pragma unroll
        for (int i = 0; i < 9; ++i) {
            c += 32 * (int64_t)limb30(i) + (neg ? -(int64_t)d.l[i] : (int64_t)d.l[i]);
            x.l[i] = i < 8 ? (int32_t)((uint32_t)c & M30) : (int32_t)c;
            c >>= 30;
        }
#pragma unroll
        for (int k = 5; k >= 0; --k) {
            N9 y;
            int64_t cy = 0;
#pragma unroll
            for (int i = 0; i < 9; ++i) {
                cy += (int64_t)x.l[i] - ((int64_t)limb30(i) << k);
                y.l[i] = i < 8 ? (int32_t)((uint32_t)cy & M30) : (int32_t)cy;
                cy >>= 30;
            }
            if (y.l[8] >= 0) x = y;
        }
        Fp r, r3;
#pragma unroll
        for (int w = 0; w < 8; ++w) {
            // bits [32 w, 32 w + 32) of x; 32 w mod 30 <= 14
            const int i = 32 * w / 30, s = 32 * w % 30;
            r.v[w] = ((uint32_t)x.l[i] >> s) | ((uint32_t)x.l[i + 1] << (30 - s));
        }
        r3.v[0] = C::R30; r3.v[1] = C::R31; r3.v[2] = C::R32; r3.v[3] = C::R33;
        r3.v[4] = C::R34; r3.v[5] = C::R35; r3.v[6] = C::R36; r3.v[7] = C::R37;
        return mul(r, r3);
    }

  private:
    struct Words {
        uint32_t v[8];
    };
    // N = (p INV + 1) / 2^32
    DV_INL static constexpr Words reduction_words() {
        const uint32_t p[8] = {C::P0, C::P1, C::P2, C::P3, C::P4, C::P5, C::P6, C::P7};
        Words r{};
        uint64_t c = 1 + (uint64_t)p[0] * C::INV;  // low word 0
        for (int i = 1; i < 8; ++i) {
            c = (c >> 32) + (uint64_t)p[i] * C::INV;
            r.v[i - 1] = (uint32_t)c;
        }
        r.v[7] = (uint32_t)(c >> 32);
        return r;
    }
    // Rows over an accumulator of four register pairs: d = x b, d += x b, d
    // += x b with the carry out added to top.
    DV_INL static void mul4(uint32_t* d, uint32_t x0, uint32_t x1, uint32_t x2, uint32_t x3, uint32_t b) {
        asm("mul.lo.u32 %0, %8, %12;\n\tmul.hi.u32 %1, %8, %12;\n\t"
            "mul.lo.u32 %2, %9, %12;\n\tmul.hi.u32 %3, %9, %12;\n\t"
            "mul.lo.u32 %4, %10, %12;\n\tmul.hi.u32 %5, %10, %12;\n\t"
            "mul.lo.u32 %6, %11, %12;\n\tmul.hi.u32 %7, %11, %12;"
            : "=&r"(d[0]), "=&r"(d[1]), "=&r"(d[2]), "=&r"(d[3]), "=&r"(d[4]), "=&r"(d[5]), "=&r"(d[6]), "=&r"(d[7])
            : "r"(x0), "r"(x1), "r"(x2), "r"(x3), "r"(b));
    }
    DV_INL static void mac4(uint32_t* d, uint32_t x0, uint32_t x1, uint32_t x2, uint32_t x3, uint32_t b) {
        asm("mad.lo.cc.u32 %0, %8, %12, %0;\n\tmadc.hi.cc.u32 %1, %8, %12, %1;\n\t"
            "madc.lo.cc.u32 %2, %9, %12, %2;\n\tmadc.hi.cc.u32 %3, %9, %12, %3;\n\t"
            "madc.lo.cc.u32 %4, %10, %12, %4;\n\tmadc.hi.cc.u32 %5, %10, %12, %5;\n\t"
            "madc.lo.cc.u32 %6, %11, %12, %6;\n\tmadc.hi.u32 %7, %11, %12, %7;"
            : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3]), "+r"(d[4]), "+r"(d[5]), "+r"(d[6]), "+r"(d[7])
            : "r"(x0), "r"(x1), "r"(x2), "r"(x3), "r"(b));
    }
    DV_INL static void mac4_top(uint32_t* d, uint32_t& top, uint32_t x0, uint32_t x1, uint32_t x2, uint32_t x3,
                                uint32_t b) {
        asm("mad.lo.cc.u32 %0, %9, %13, %0;\n\tmadc.hi.cc.u32 %1, %9, %13, %1;\n\t"
            "madc.lo.cc.u32 %2, %10, %13, %2;\n\tmadc.hi.cc.u32 %3, %10, %13, %3;\n\t"
            "madc.lo.cc.u32 %4, %11, %13, %4;\n\tmadc.hi.cc.u32 %5, %11, %13, %5;\n\t"
            "madc.lo.cc.u32 %6, %12, %13, %6;\n\tmadc.hi.cc.u32 %7, %12, %13, %7;\n\t"
            "addc.u32 %8, %8, 0;"
            : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3]), "+r"(d[4]), "+r"(d[5]), "+r"(d[6]), "+r"(d[7]),
              "+r"(top)
            : "r"(x0), "r"(x1), "r"(x2), "r"(x3), "r"(b));
    }
    // The shift of T = E + 2^32 O by one limb (the low limb is done with): o
    // becomes the new E with e[1] added to its low word, whose carry (the
    // weight of the new O's low word) starts the chain t = x b + (e without two words).
    DV_INL static void shift_mac4(uint32_t* t, uint32_t* o, const uint32_t* e, uint32_t x0, uint32_t x1, uint32_t x2,
                                  uint32_t x3, uint32_t b) {
        asm("add.cc.u32 %8, %8, %14;\n\t"
            "madc.lo.cc.u32 %0, %9, %13, %15;\n\tmadc.hi.cc.u32 %1, %9, %13, %16;\n\t"
            "madc.lo.cc.u32 %2, %10, %13, %17;\n\tmadc.hi.cc.u32 %3, %10, %13, %18;\n\t"
            "madc.lo.cc.u32 %4, %11, %13, %19;\n\tmadc.hi.cc.u32 %5, %11, %13, %20;\n\t"
            "madc.lo.cc.u32 %6, %12, %13, 0;\n\tmadc.hi.u32 %7, %12, %13, 0;"
            : "=&r"(t[0]), "=&r"(t[1]), "=&r"(t[2]), "=&r"(t[3]), "=&r"(t[4]), "=&r"(t[5]), "=&r"(t[6]), "=&r"(t[7]),
              "+r"(o[0])
            : "r"(x0), "r"(x1), "r"(x2), "r"(x3), "r"(b), "r"(e[1]), "r"(e[2]), "r"(e[3]), "r"(e[4]), "r"(e[5]),
              "r"(e[6]), "r"(e[7]));
    }
    DV_INL static void rotate(uint32_t* e, uint32_t* o, const uint32_t* t) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            e[j] = o[j];
            o[j] = t[j];
        }
    }
    // One step with the exact multiplier: afterwards e[0] = 0.
    DV_INL static void reduce_step(uint32_t* e, uint32_t* o) {
        const uint32_t m = e[0] * C::INV;
        mac4(o, C::P1, C::P3, C::P5, C::P7, m);
        mac4_top(e, o[7], C::P0, C::P2, C::P4, C::P6, m);
    }
    // r = (E >> 32) + O
    DV_INL static void merge(uint32_t* r, const uint32_t* e, const uint32_t* o) {
        asm("add.cc.u32 %0, %8, %16;\n\taddc.cc.u32 %1, %9, %17;\n\taddc.cc.u32 %2, %10, %18;\n\t"
            "addc.cc.u32 %3, %11, %19;\n\taddc.cc.u32 %4, %12, %20;\n\taddc.cc.u32 %5, %13, %21;\n\t"
            "addc.cc.u32 %6, %14, %22;\n\taddc.u32 %7, %15, 0;"
            : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3]), "=&r"(r[4]), "=&r"(r[5]), "=&r"(r[6]), "=&r"(r[7])
            : "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7]), "r"(e[1]),
              "r"(e[2]), "r"(e[3]), "r"(e[4]), "r"(e[5]), "r"(e[6]), "r"(e[7]));
    }
    // K products x[k] m added to the pairs at d, the carry out to top.
    template <int K>
    DV_INL static void chain(uint32_t* d, const uint32_t* x, uint32_t m, uint32_t& top) {
        if constexpr (K == 1)
            asm("mad.lo.cc.u32 %0, %3, %4, %0;\n\tmadc.hi.cc.u32 %1, %3, %4, %1;\n\taddc.u32 %2, %2, 0;"
                : "+r"(d[0]), "+r"(d[1]), "+r"(top)
                : "r"(x[0]), "r"(m));
        else if constexpr (K == 2)
            asm("mad.lo.cc.u32 %0, %5, %7, %0;\n\tmadc.hi.cc.u32 %1, %5, %7, %1;\n\t"
                "madc.lo.cc.u32 %2, %6, %7, %2;\n\tmadc.hi.cc.u32 %3, %6, %7, %3;\n\taddc.u32 %4, %4, 0;"
                : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3]), "+r"(top)
                : "r"(x[0]), "r"(x[1]), "r"(m));
        else if constexpr (K == 3)
            asm("mad.lo.cc.u32 %0, %7, %10, %0;\n\tmadc.hi.cc.u32 %1, %7, %10, %1;\n\t"
                "madc.lo.cc.u32 %2, %8, %10, %2;\n\tmadc.hi.cc.u32 %3, %8, %10, %3;\n\t"
                "madc.lo.cc.u32 %4, %9, %10, %4;\n\tmadc.hi.cc.u32 %5, %9, %10, %5;\n\taddc.u32 %6, %6, 0;"
                : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3]), "+r"(d[4]), "+r"(d[5]), "+r"(top)
                : "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(m));
        else
            mac4_top(d, top, x[0], x[1], x[2], x[3], m);
    }
    // E + 2^32 O of a 512-bit value
    DV_INL static Wide combine(const uint32_t* e, const uint32_t* o) {
        Wide a, b;
        b.v[0] = 0;
#pragma unroll
        for (int j = 0; j < 16; ++j) a.v[j] = e[j];
#pragma unroll
        for (int j = 1; j < 16; ++j) b.v[j] = o[j - 1];
        return wide_add(a, b);
    }
    // Signed 30-bit-limb numbers of the divstep inverse.
    struct N9 {
        int32_t l[9];
        DV_INL bool nonzero() const {
            int32_t o = 0;
#pragma unroll
            for (int i = 0; i < 9; ++i) o |= l[i];
            return o != 0;
        }
    };
    // bits [30 i, 30 i + 30) of p and of a
    DV_INL static constexpr int32_t limb30(int i) {
        const uint32_t p[8] = {C::P0, C::P1, C::P2, C::P3, C::P4, C::P5, C::P6, C::P7};
        const int b = 30 * i, w = b >> 5, s = b & 31;
        const uint32_t lo = p[w] >> s, hi = (s > 2 && w + 1 < 8) ? p[w + 1] << (32 - s) : 0u;
        return (int32_t)((lo | hi) & ((1u << 30) - 1));
    }
    DV_INL static uint32_t bits30(const Fp& a, int i) {
        const int b = 30 * i, w = b >> 5, s = b & 31;
        uint32_t x = a.v[w] >> s;
        if (s > 2 && w + 1 < 8) x |= a.v[w + 1] << (32 - s);
        return x & ((1u << 30) - 1);
    }
    // 30 divsteps on the low bits of f and g (f odd): delta and the matrix
    // t = (u, v, q, r) with t (f, g) = 2^30 (f', g').  A step with g odd and
    // delta > 0 swaps first: (f, g) <- (g, -f), (u, v, q, r) <- (q, r, -u, -v),
    // delta <- -delta; then g odd adds f to g and (u, v) to (q, r); then g
    // halves, (u, v) double and delta grows by one.
    DV_INL static int divsteps30(int delta, uint32_t f, uint32_t g, int32_t* t) {
        int32_t u = 1, v = 0, q = 0, r = 1;
#pragma unroll
        for (int i = 0; i < 30; ++i) {
            const bool odd = g & 1u, swap = odd && delta > 0;
            const uint32_t f1 = swap ? g : f, g1 = swap ? 0u - f : g;
            const int32_t u1 = swap ? q : u, v1 = swap ? r : v, q1 = swap ? -u : q, r1 = swap ? -v : r;
            delta = swap ? -delta : delta;
            f = f1;
            g = (odd ? g1 + f1 : g1) >> 1;
            q = odd ? q1 + u1 : q1;
            r = odd ? r1 + v1 : r1;
            u = 2 * u1;
            v = 2 * v1;
            ++delta;
        }
        t[0] = u;
        t[1] = v;
        t[2] = q;
        t[3] = r;
        return delta;
    }
};

typedef Fp<FqCfg> Fq;
typedef Fp<FrCfg> Fr;

// Fq2 = Fq[u] / (u^2 + 1)
struct Fq2 {
    Fq c0, c1;
    DV_INL static Fq2 zero() { return {Fq::zero(), Fq::zero()}; }
    DV_INL static Fq2 one() { return {Fq::one(), Fq::zero()}; }
    DV_INL bool is_zero() const { return c0.is_zero() && c1.is_zero(); }
    DV_INL bool operator==(const Fq2& o) const { return c0 == o.c0 && c1 == o.c1; }
    DV_INL static Fq2 add(const Fq2& a, const Fq2& b) { return {Fq::add(a.c0, b.c0), Fq::add(a.c1, b.c1)}; }
    DV_INL static Fq2 sub(const Fq2& a, const Fq2& b) { return {Fq::sub(a.c0, b.c0), Fq::sub(a.c1, b.c1)}; }
    DV_INL static Fq2 dbl(const Fq2& a) { return {Fq::dbl(a.c0), Fq::dbl(a.c1)}; }
    DV_INL static Fq2 neg(const Fq2& a) { return {Fq::neg(a.c0), Fq::neg(a.c1)}; }
    DV_INL static Fq2 conj(const Fq2& a) { return {a.c0, Fq::neg(a.c1)}; }
    // Products keep the three Karatsuba products at 512 bits and reduce twice
    // (336 multiply-adds against 408 with each product reduced), in one
    // out-of-line body each: a call moves its operands once.
    __device__ __noinline__ static Fq2 mul(Fq2 a, Fq2 b) {
        const Fq::Wide t0 = Fq::mul_wide(a.c0, b.c0), t1 = Fq::mul_wide(a.c1, b.c1);
        const Fq::Wide t2 = Fq::mul_wide(Fq::add_raw(a.c0, a.c1), Fq::add_raw(b.c0, b.c1));
        const Fq c1 = Fq::redc(Fq::wide_sub(t2, Fq::wide_add(t0, t1)));  // < 2 p^2
        Fq::Wide d = Fq::wide_sub(t0, t1);
        Fq::make_positive(d);
        return {Fq::redc(d), c1};
    }
    // (c0 + c1 u)^2 = (c0+c1)(c0-c1) + 2 c0 c1 u
    __device__ __noinline__ static Fq2 sqr(Fq2 a) {
        const Fq m = Fq::mul_inl(Fq::add_raw(a.c0, a.c1), Fq::sub(a.c0, a.c1));
        return {m, Fq::dbl(Fq::mul_inl(a.c0, a.c1))};
    }
    // a b - c d: six products, two reductions (528 multiply-adds against 672)
    __device__ __noinline__ static Fq2 mul_sub(Fq2 a, Fq2 b, Fq2 c, Fq2 d) {
        Fq::Wide w = Fq::mul_wide(a.c0, b.c0), x = w, y = w;
        w = Fq::mul_wide(a.c1, b.c1);
        x = Fq::wide_sub(x, w);
        y = Fq::wide_sub(Fq::mul_wide(Fq::add_raw(a.c0, a.c1), Fq::add_raw(b.c0, b.c1)), Fq::wide_add(y, w));
        w = Fq::mul_wide(c.c0, d.c0);
        x = Fq::wide_sub(x, w);
        y = Fq::wide_add(y, w);
        w = Fq::mul_wide(c.c1, d.c1);
        x = Fq::wide_add(x, w);
        y = Fq::wide_add(y, w);
        y = Fq::wide_sub(y, Fq::mul_wide(Fq::add_raw(c.c0, c.c1), Fq::add_raw(d.c0, d.c1)));
        Fq::make_positive(x);
        Fq::make_positive(y);
        return {Fq::redc(x), Fq::redc(y)};
    }
    DV_INL static Fq2 mul_fq(const Fq2& a, const Fq& s) { return {Fq::mul(a.c0, s), Fq::mul(a.c1, s)}; }
    DV_INL static Fq2 inv(const Fq2& a) {
        const Fq n = Fq::add(Fq::sqr(a.c0), Fq::sqr(a.c1));
        const Fq ni = Fq::inv(n);
        return {Fq::mul(a.c0, ni), Fq::neg(Fq::mul(a.c1, ni))};
    }
};

}  // namespace dv
