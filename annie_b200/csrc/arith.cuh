// Device arithmetic of the modular-squaring engine (sm_100a).
//
// Two prime sets.
// * The transform primes (this engine's own choice): six primes p < 2^30 with
//   2^23 | p - 1.  A value mod p is kept lazily in [0, 2p) or [0, 4p) (4p <
//   2^32), so the NTT butterflies need no full reduction (Harvey's lazy
//   butterflies): a forward butterfly is a Shoup product (x w mod p with the
//   precomputed w' = floor(w 2^32 / p): 1 mulhi + 2 mul) and three adds.  A
//   class of the reference with K primes uses K + 1 of them: their product
//   exceeds the reference's prime product for every K, so every convolution
//   the reference computes exactly is exact here too.
// * The reference's primes (src/transformGPU.h:79-83, p in (2^31, 2^32)) are
//   only used to convert registers to and from the reference's register words
//   (its normal form is the residues, mod these primes, of each coefficient's
//   exact value; ocl/kernel.cl:1476-1559).
//
// A register's normal form is held as each coefficient's exact value: a
// 96-bit two's-complement integer in three 32-bit limbs.
#pragma once
#include <cstdint>

typedef uint32_t u32;
typedef uint64_t u64;
typedef int32_t i32;
typedef int64_t i64;

#define AB_MAXK 5          // primes of the reference's largest class
#define AB_MAXKP 6         // transform primes of that class
#define AB_NW 3            // words of a coefficient's exact value

// ---------------------------------------------------------------- transform primes
// x in [0, 4p) -> [0, 2p); p2 = 2p.  (x - 2p wraps above x when x < 2p.)
__device__ __forceinline__ u32 red2(u32 x, u32 p2) { return min(x, x - p2); }

// x w mod p in [0, 2p) for any x < 2^32 (Shoup: ws = floor(w 2^32 / p), w < p)
__device__ __forceinline__ u32 shoup(u32 x, u32 w, u32 ws, u32 p)
{
	const u32 q = __umulhi(x, ws);
	return x * w - q * p;
}

// t 2^-32 mod p for a 64-bit t < f 2^32 p, in (0, (f + 1) p) (Montgomery,
// pinv = p^-1 mod 2^32).
__device__ __forceinline__ u32 redc(u64 t, u32 p, u32 pinv)
{
	return (u32)(t >> 32) - __umulhi((u32)t * pinv, p) + p;
}

// w 2^32 mod p from the Shoup pair (w, floor(w 2^32 / p)) of w
__device__ __forceinline__ u32 mont_twiddle(uint2 w, u32 p) { return 0u - w.y * p; }

// (x0 + x1 X)(y0 + y1 X) 2^-32 mod (X^2 - c), in place in (x0, x1); words in
// [0, 2p) (in and out), cm = c 2^32 mod p.  Products are summed in 64 bits
// before their one reduction (below 2^32 2p: x y < 4 p^2 and p < 2^30), three
// reductions for the four products and the twiddle.  Without mul, y = x.
__device__ __forceinline__ void poly_product(u32 & x0, u32 & x1, u32 y0, u32 y1, bool mul, u32 cm, u32 p, u32 p2, u32 pinv)
{
	const u32 t = redc((u64)x1 * y1, p, pinv);
	const u32 r0 = redc((u64)x0 * y0 + (u64)t * cm, p, pinv);
	const u32 r1 = mul ? redc((u64)x0 * y1 + (u64)x1 * y0, p, pinv) : redc((u64)(x0 + x0) * x1, p, pinv);
	x0 = red2(r0, p2);
	x1 = red2(r1, p2);
}

// Forward (decimation-in-time form) butterfly x0 +- w x1, inputs and outputs
// in [0, 4p).
__device__ __forceinline__ void fwd_bf(u32 & x0, u32 & x1, u32 w, u32 ws, u32 p, u32 p2)
{
	const u32 a = red2(x0, p2);
	const u32 t = shoup(x1, w, ws, p);
	x0 = a + t;
	x1 = a - t + p2;
}

// Inverse (Gentleman-Sande) butterfly with the stored twiddle v = -w^-1:
// x0 + x1 and (x1 - x0) v = (x0 - x1) w^-1; inputs and outputs in [0, 2p).
__device__ __forceinline__ void inv_bf(u32 & x0, u32 & x1, u32 v, u32 vs, u32 p, u32 p2)
{
	const u32 s = x0 + x1, d = x1 - x0 + p2;
	x0 = red2(s, p2);
	x1 = shoup(d, v, vs, p);
}

// ---------------------------------------------------------------- constants
// Per-transform constants, passed by value to every kernel (kernel-parameter
// constant bank).
struct TConst
{
	u32 p[AB_MAXKP], pinv[AB_MAXKP];
	u32 enc[AB_MAXKP][3];                // s_k 2^(32 j) 2^32 mod p: encoding weights of a value's limbs (encode_res)
	u32 mk[AB_MAXKP][AB_MAXK];           // e_k M/p_k in radix 2^30, the top entry holding 32 bits (crt)
	u32 mkh[AB_MAXKP];                   // bits above those 32
	u32 negm[AB_MAXK], negmh;            // -M mod 2^(32 K) in the same form
	u32 tinv, tsh;                       // quotient estimate of crt: 2^tsh 2^(32 + 30 (K-1)) / M, times 2^32
	int K, KP, pck, lbase, ln;           // reference primes K, transform primes KP = K + 1
	u32 n;                               // 2^ln
	u32 R, H;                            // column pass: row length and row count of the 2-D layout
	u32 HR;                              // row pass: rows (H 2^G) of 2^(LB+1) words
	int LA, LB, G;                       // column levels, row levels, mid levels (lengths above 2^20)
};

// N as a sparse polynomial: its nonzero coefficients, when there are at most
// AB_SPARSE of them (k 2^m + 1 has two or three: 1, and k across one or two
// coefficients).
#define AB_SPARSE 3
struct SparseN
{
	u32 nt;                              // 0: N is dense
	u32 idx[AB_SPARSE];
	u32 coef[AB_SPARSE][AB_NW];
};

// Digit size and modulus of one candidate (candidates of a batch share K and
// the length).
struct CandConst
{
	int lbase;
	SparseN sp;
};

// ---------------------------------------------------------------- big ints
template <int L>
struct Big
{
	u32 l[L];
};

template <int L>
__device__ __forceinline__ Big<L> big_zero()
{
	Big<L> r;
#pragma unroll
	for (int i = 0; i < L; ++i) r.l[i] = 0;
	return r;
}

// a + b + carry-in chain; the carry flag lives only inside one asm statement,
// so each chain is one statement.
template <int L>
__device__ __forceinline__ Big<L> big_add(const Big<L> & a, const Big<L> & b)
{
	static_assert(L >= 2 && L <= 5, "2 to 5 limbs");
	Big<L> r;
	if constexpr (L == 2)
		asm("add.cc.u32 %0, %2, %4;\n\taddc.u32 %1, %3, %5;"
		    : "=&r"(r.l[0]), "=r"(r.l[1]) : "r"(a.l[0]), "r"(a.l[1]), "r"(b.l[0]), "r"(b.l[1]));
	else if constexpr (L == 3)
		asm("add.cc.u32 %0, %3, %6;\n\taddc.cc.u32 %1, %4, %7;\n\taddc.u32 %2, %5, %8;"
		    : "=&r"(r.l[0]), "=&r"(r.l[1]), "=r"(r.l[2])
		    : "r"(a.l[0]), "r"(a.l[1]), "r"(a.l[2]), "r"(b.l[0]), "r"(b.l[1]), "r"(b.l[2]));
	else if constexpr (L == 4)
		asm("add.cc.u32 %0, %4, %8;\n\taddc.cc.u32 %1, %5, %9;\n\taddc.cc.u32 %2, %6, %10;\n\taddc.u32 %3, %7, %11;"
		    : "=&r"(r.l[0]), "=&r"(r.l[1]), "=&r"(r.l[2]), "=r"(r.l[3])
		    : "r"(a.l[0]), "r"(a.l[1]), "r"(a.l[2]), "r"(a.l[3]), "r"(b.l[0]), "r"(b.l[1]), "r"(b.l[2]), "r"(b.l[3]));
	else
		asm("add.cc.u32 %0, %5, %10;\n\taddc.cc.u32 %1, %6, %11;\n\taddc.cc.u32 %2, %7, %12;\n\taddc.cc.u32 %3, %8, %13;\n\t"
		    "addc.u32 %4, %9, %14;"
		    : "=&r"(r.l[0]), "=&r"(r.l[1]), "=&r"(r.l[2]), "=&r"(r.l[3]), "=r"(r.l[L - 1])
		    : "r"(a.l[0]), "r"(a.l[1]), "r"(a.l[2]), "r"(a.l[3]), "r"(a.l[L - 1]),
		      "r"(b.l[0]), "r"(b.l[1]), "r"(b.l[2]), "r"(b.l[3]), "r"(b.l[L - 1]));
	return r;
}

template <int L>
__device__ __forceinline__ Big<L> big_sub(const Big<L> & a, const Big<L> & b)
{
	static_assert(L >= 2 && L <= 5, "2 to 5 limbs");
	Big<L> r;
	if constexpr (L == 2)
		asm("sub.cc.u32 %0, %2, %4;\n\tsubc.u32 %1, %3, %5;"
		    : "=&r"(r.l[0]), "=r"(r.l[1]) : "r"(a.l[0]), "r"(a.l[1]), "r"(b.l[0]), "r"(b.l[1]));
	else if constexpr (L == 3)
		asm("sub.cc.u32 %0, %3, %6;\n\tsubc.cc.u32 %1, %4, %7;\n\tsubc.u32 %2, %5, %8;"
		    : "=&r"(r.l[0]), "=&r"(r.l[1]), "=r"(r.l[2])
		    : "r"(a.l[0]), "r"(a.l[1]), "r"(a.l[2]), "r"(b.l[0]), "r"(b.l[1]), "r"(b.l[2]));
	else if constexpr (L == 4)
		asm("sub.cc.u32 %0, %4, %8;\n\tsubc.cc.u32 %1, %5, %9;\n\tsubc.cc.u32 %2, %6, %10;\n\tsubc.u32 %3, %7, %11;"
		    : "=&r"(r.l[0]), "=&r"(r.l[1]), "=&r"(r.l[2]), "=r"(r.l[3])
		    : "r"(a.l[0]), "r"(a.l[1]), "r"(a.l[2]), "r"(a.l[3]), "r"(b.l[0]), "r"(b.l[1]), "r"(b.l[2]), "r"(b.l[3]));
	else
		asm("sub.cc.u32 %0, %5, %10;\n\tsubc.cc.u32 %1, %6, %11;\n\tsubc.cc.u32 %2, %7, %12;\n\tsubc.cc.u32 %3, %8, %13;\n\t"
		    "subc.u32 %4, %9, %14;"
		    : "=&r"(r.l[0]), "=&r"(r.l[1]), "=&r"(r.l[2]), "=&r"(r.l[3]), "=r"(r.l[L - 1])
		    : "r"(a.l[0]), "r"(a.l[1]), "r"(a.l[2]), "r"(a.l[3]), "r"(a.l[L - 1]),
		      "r"(b.l[0]), "r"(b.l[1]), "r"(b.l[2]), "r"(b.l[3]), "r"(b.l[L - 1]));
	return r;
}

template <int L>
__device__ __forceinline__ Big<L> big_neg(const Big<L> & a) { return big_sub<L>(big_zero<L>(), a); }

template <int L>
__device__ __forceinline__ Big<L> big_add_u32(const Big<L> & a, u32 v)
{
	Big<L> r;
	u64 c = v;
#pragma unroll
	for (int i = 0; i < L; ++i) { c += a.l[i]; r.l[i] = (u32)c; c >>= 32; }
	return r;
}

// a * y mod 2^(32L), y unsigned (sign-agnostic two's-complement product)
template <int L>
__device__ __forceinline__ Big<L> big_mul_u32(const Big<L> & a, u32 y)
{
	Big<L> r;
	u64 c = 0;
#pragma unroll
	for (int i = 0; i < L; ++i) { c += (u64)a.l[i] * y; r.l[i] = (u32)c; c >>= 32; }
	return r;
}

template <int L>
__device__ __forceinline__ bool big_is_neg(const Big<L> & a) { return (a.l[L - 1] >> 31) != 0; }

// a 96-bit exact value (three limbs) sign-extended or truncated to L limbs
template <int L>
__device__ __forceinline__ Big<L> big_from_exact(u32 d0, u32 d1, u32 d2)
{
	Big<L> r;
	const u32 s = ((i32)d2 < 0) ? 0xffffffffu : 0u;
#pragma unroll
	for (int i = 0; i < L; ++i) r.l[i] = (i == 0) ? d0 : (i == 1) ? d1 : (i == 2) ? d2 : s;
	return r;
}

// ---------------------------------------------------------------- CRT
// Every forward image carries a factor s_k per prime (encode_res), chosen so
// that the inverse output of a product, (n/2) 2^-32 s_k^2 V mod p_k, is already
// the CRT coordinate of V: s_k^2 e_k = (2/n) 2^32 (M/p_k)^-1 mod p_k, with e_k
// = 1, or the least non-residue mod p_k when that quotient is not a square.
// So V = sum y_k e_k (M/p_k) - t M for ANY representative y_k of the inverse
// output (here [0, 2p_k), as the lazy levels leave it): no product and no
// reduction per residue.  t = round(S / M), S the sum: S / M lies within
// |V| / M < 2^-18 of the integer t, so its top 32 bits decide t.
//
// S is summed in radix 2^30, one 64-bit column per limb: the integer
// multiplier is what bounds the column pass (B200: IMAD 64, IMAD.HI and
// IMAD.WIDE 32 per clock and SM), and 2^31 2^30 products of 6 primes fit a
// column with no carry chain, so a limb product costs one IMAD.WIDE (2 units)
// where a 32-bit limb costs a low and a high product (3).  Computed mod
// 2^(32 L), where V fits.
template <int L>
__device__ __forceinline__ Big<L> crt(const TConst & c, const u32 (&y)[L + 1])
{
	constexpr int KP = L + 1;
	u64 col[L];
#pragma unroll
	for (int j = 0; j < L; ++j)
	{
		u64 s = (u64)y[0] * c.mk[0][j];
#pragma unroll
		for (int k = 1; k < KP; ++k) s += (u64)y[k] * c.mk[k][j];
		col[j] = s;
	}
	// only e_3 = 11 of the class L = 4 needs a 33rd bit
	if (L == 4) col[L - 1] += (u64)(y[3] * c.mkh[3]) << 32;
	const u32 hi = (u32)((col[L - 1] + (col[L - 2] >> 30)) >> 32);
	const u32 t = (__umulhi(hi, c.tinv) + (1u << (c.tsh - 1))) >> c.tsh;
#pragma unroll
	for (int j = 0; j < L; ++j) col[j] += (u64)t * c.negm[j];
	col[L - 1] += (u64)(t * c.negmh) << 32;
#pragma unroll
	for (int j = 1; j < L; ++j) col[j] += col[j - 1] >> 30;
	Big<L> V;
#pragma unroll
	for (int i = 0; i < L - 1; ++i) V.l[i] = __funnelshift_r((u32)col[i] << 2, (u32)col[i + 1], 2 + 2 * i);
	V.l[L - 1] = (u32)(col[L - 1] >> (2 * (L - 1)));
	return V;
}

// Coefficient e of N(x) m(x) mod x^n + 1, mod 2^(32 L), for a sparse N;
// get(i, d0, d1, d2) reads the exact value m_i.
template <int L, typename Get>
__device__ __forceinline__ Big<L> sparse_product(const SparseN & s, u32 e, u32 n, Get get)
{
	Big<L> v = big_zero<L>();
	const u32 nt = s.nt;
	for (u32 t = 0; t < nt; ++t)
	{
		const u32 i = s.idx[t];
		u32 d0, d1, d2;
		get((e - i) & (n - 1), d0, d1, d2);
		Big<L> m = big_from_exact<L>(d0, d1, d2);
		if (e < i) m = big_neg<L>(m);
#pragma unroll
		for (int j = 0; j < AB_NW && j < L; ++j)
		{
			const u32 q = s.coef[t][j];
			if (q == 0u) continue;           // the same in every thread
			const Big<L> x = (q == 1u) ? m : big_mul_u32<L>(m, q);
			Big<L> y;
#pragma unroll
			for (int l = 0; l < L; ++l) y.l[l] = (l < j) ? 0u : x.l[(l - j + L) % L];
			v = big_add<L>(v, y);
		}
	}
	return v;
}

// s_k v mod p_k in (0, 4p) for any exact value v (three limbs): one Montgomery
// reduction of the 64-bit sum of the weighted limbs, the top one signed.  The
// sign of s_k is chosen so that enc[0] + enc[1] + enc[2] / 2 <= 2p
// (encode_weights), so the sum's high word lies in [-p/2, 2p).
__device__ __forceinline__ u32 encode_res(const TConst & c, int k, u32 d0, u32 d1, u32 d2)
{
	const u32 p = c.p[k];
	u64 s = (u64)d0 * c.enc[k][0];
	s += (u64)d1 * c.enc[k][1];
	s += (u64)((i64)(i32)d2 * (i32)c.enc[k][2]);
	return (u32)(s >> 32) - __umulhi((u32)s * c.pinv[k], p) + 2 * p;
}

// ---------------------------------------------------------------- digits
// A coefficient is pck digits of lbase bits; the carry rule (unsigned digits,
// the top one balanced; ocl/kernel.cl:1478-1537) only depends on the
// coefficient as one digit of W = pck lbase bits, W = 32 ws + bs.  W is the
// same in every thread, so the limb moves are uniform branches.
struct Width
{
	int ws, bs;
	u32 mask;                            // low bs bits
};
__device__ __forceinline__ Width make_width(int w)
{
	return Width{ w >> 5, w & 31, (1u << (w & 31)) - 1 };
}

// Limbs that hold W bits: lbase <= 31, pck lbase <= 80.
template <int PCK>
struct DigitLimbs { static constexpr int N = (PCK == 1) ? 1 : (PCK == 2) ? 2 : 3; };

// d = the low W bits of f (unsigned), f >>= W (arithmetic).  FULL: W reaches
// into the last of the ND limbs (ws = ND - 1), as the digit sizes of the
// parameter rule do for bases up to 100; smaller sizes (larger bases, forced
// parameters) take the general form.
template <bool FULL, int L, int ND>
__device__ __forceinline__ void split_digit(Big<L> & f, const Width & w, u32 (&d)[ND])
{
	const u32 fill = (u32)((i32)f.l[L - 1] >> 31);
	u32 t[L + ND];
#pragma unroll
	for (int i = 0; i < L + ND; ++i) t[i] = (i < L) ? f.l[i % L] : fill;
	if constexpr (FULL)
	{
#pragma unroll
		for (int i = 0; i < ND; ++i) d[i] = (i < ND - 1) ? t[i] : t[i] & w.mask;
#pragma unroll
		for (int i = 0; i < L; ++i) f.l[i] = (i + ND - 1 < L) ? __funnelshift_r(t[i + ND - 1], t[i + ND], w.bs) : fill;
	}
	else
	{
#pragma unroll
		for (int i = 0; i < ND; ++i) d[i] = (i < w.ws) ? t[i] : (i == w.ws) ? t[i] & w.mask : 0u;
		for (int m = 0; m < w.ws; ++m)
		{
#pragma unroll
			for (int i = 0; i < L; ++i) t[i] = t[i + 1];
		}
#pragma unroll
		for (int i = 0; i < L; ++i) f.l[i] = __funnelshift_r(t[i], t[i + 1], w.bs);
	}
}

// f + d (d unsigned)
template <int L, int ND>
__device__ __forceinline__ Big<L> add_digit(const Big<L> & f, const u32 (&d)[ND])
{
	Big<L> t;
#pragma unroll
	for (int i = 0; i < L; ++i) t.l[i] = (i < ND) ? d[i % ND] : 0u;
	return big_add<L>(f, t);
}

// ---------------------------------------------------------------- reference primes
// Montgomery arithmetic mod the reference's primes (p in (2^31, 2^32),
// canonical results; src/transformGPU.h:21-59), for the register-word
// conversions only.
struct RefConst
{
	u32 p[AB_MAXK], q[AB_MAXK];          // q = p^-1 mod 2^32
	u32 r2[AB_MAXK];                     // 2^64 mod p (Montgomery form of 2^32)
	u32 gm[AB_MAXK][AB_MAXK], gmq[AB_MAXK][AB_MAXK];   // Montgomery form of P_j^-1 mod P_i (j > i), and * q_i
	int K;
};

__device__ __forceinline__ u32 ref_sub(u32 a, u32 b, u32 p)
{
	const u32 d = a - b;
	return (a < b) ? d + p : d;
}

__device__ __forceinline__ u32 ref_mont_c(u32 a, u32 w, u32 wq, u32 p)
{
	return ref_sub(__umulhi(a, w), __umulhi(a * wq, p), p);
}

// x mod p, any u32 x (p > 2^31)
__device__ __forceinline__ u32 ref_red(u32 x, u32 p) { return (x >= p) ? x - p : x; }
