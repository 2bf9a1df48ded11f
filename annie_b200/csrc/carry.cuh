// The carry of one group of 4 coefficients by 4 adjacent lanes, a lane per
// coefficient (j = 0..3 its place).  One thread per group does the same with
// fewer instructions (columns.cuh); the lanes shorten the chain of dependent
// ones to about a third, which is what bounds a launch too small to fill the
// GPU.  All lanes of a warp call these together.
#pragma once
#include "arith.cuh"

namespace ab
{

// The lane's value from the lane below (NC limbs passed, sign-extended to L).
template <int L, int NC>
__device__ __forceinline__ Big<L> shfl_up4(const Big<L> & a)
{
	Big<L> r;
#pragma unroll
	for (int i = 0; i < L; ++i) r.l[i] = (i < NC) ? __shfl_up_sync(0xffffffffu, a.l[i], 1, 4) : (u32)((i32)r.l[NC - 1] >> 31);
	return r;
}

// Phase 1: f = the lane's exact product coefficient on entry; d = its unsigned
// W-bit digit; on return lane 3's f is the group's carry-out.
template <bool FULL, int L, int ND>
__device__ __forceinline__ void lane_digits(Big<L> & f, const Width & w, u32 j, u32 (&d)[ND])
{
	constexpr int NC = FULL ? L - ND + 1 : L;        // limbs of f >> W
#pragma unroll
	for (int r = 1; r < 4; ++r)
	{
		Big<L> h = f;
		split_digit<FULL, L, ND>(h, w, d);
		const Big<L> up = shfl_up4<L, NC>(h);
		if (j == (u32)r) f = big_add<L>(f, up);
	}
	split_digit<FULL, L, ND>(f, w, d);
}

// Limbs that hold every sum of phase 2.  The carry into the second coefficient
// of a group is below 2^(32 L - 1 - 2 W) in magnitude: with FULL (W >= 32 (ND - 1))
// below 2^63, so two limbs pass it on and three hold the sums; other digit sizes
// take all L.
template <bool FULL, int L>
struct CarryLimbs
{
	static constexpr int N = (FULL || L < AB_NW) ? AB_NW : L, PASS = FULL ? 2 : N;
};

// v as a sum of phase 2 (sign-extended)
template <int CL, int L>
__device__ __forceinline__ Big<CL> carry_extend(const Big<L> & v)
{
	Big<CL> r;
#pragma unroll
	for (int i = 0; i < CL; ++i) r.l[i] = (i < L) ? v.l[i % L] : (u32)((i32)v.l[L - 1] >> 31);
	return r;
}

// Phase 2: cin = the previous group's carry-out (lane 0; 0 in the others), d =
// the digits; x = the exact value: balanced in lanes 0..2, lane 3 absorbs the
// rest.  half: 2^(W-1).
template <bool FULL, int L, int ND>
__device__ __forceinline__ void lane_balance(const Big<L> & cin, const u32 (&d)[ND], const Width & w, const Big<AB_NW> & half, u32 j, u32 (&x)[AB_NW])
{
	constexpr int CL = CarryLimbs<FULL, L>::N;
	u32 hd[ND], dd[ND];
#pragma unroll
	for (int i = 0; i < ND; ++i) hd[i] = half.l[i];
	Big<L> v = add_digit<L, ND>(add_digit<L, ND>(cin, d), hd);
	split_digit<FULL, L, ND>(v, w, dd);
	Big<CL> c = carry_extend<CL, L>(v), t;
#pragma unroll
	for (int i = 0; i < CL; ++i) t.l[i] = (i < ND) ? d[i % ND] : 0u;
#pragma unroll
	for (int r = 1; r < 4; ++r)
	{
		const Big<CL> up = shfl_up4<CL, CarryLimbs<FULL, L>::PASS>(c);
		if (j == (u32)r) t = big_add<CL>(t, up);
		if (r < 3)
		{
			u32 e[ND];
			c = big_add<CL>(t, carry_extend<CL, AB_NW>(half));
			split_digit<FULL, CL, ND>(c, w, e);
			if (j == (u32)r)
			{
#pragma unroll
				for (int i = 0; i < ND; ++i) dd[i] = e[i];
			}
		}
	}
	Big<AB_NW> b;
#pragma unroll
	for (int i = 0; i < AB_NW; ++i) b.l[i] = (i < ND) ? dd[i % ND] : 0u;
	b = big_sub<AB_NW>(b, half);
#pragma unroll
	for (int i = 0; i < AB_NW; ++i) x[i] = (j < 3) ? b.l[i] : t.l[i];
}

// 2^(W-1) as three limbs
__device__ __forceinline__ Big<AB_NW> half_of(int wbits)
{
	const int hb = wbits - 1;
	Big<AB_NW> h;
#pragma unroll
	for (int i = 0; i < AB_NW; ++i) h.l[i] = (i == (hb >> 5)) ? 1u << (hb & 31) : 0u;
	return h;
}

// x >= 2^W (exact value, signed)
__device__ __forceinline__ bool reaches_width(const u32 (&x)[AB_NW], const Width & w)
{
	Big<AB_NW> t;
#pragma unroll
	for (int i = 0; i < AB_NW; ++i) t.l[i] = x[i];
	u32 e[AB_NW];
	split_digit<false, AB_NW, AB_NW>(t, w, e);
	return (i32)t.l[2] >= 0 && (t.l[0] | t.l[1] | t.l[2]) != 0u;
}

} // namespace ab
