// Butterfly levels of a transform of 2^LN words held in shared memory
// (resident.cuh).
//
// 8 words per thread: stages of 3 levels, the top one taking the remainder,
// and a bottom step of two levels, the pointwise product and two inverse
// levels.  A stage costs a shared-memory round trip and a barrier, about the
// same as its three levels; 16 words per thread would save one stage, but
// halves the warps that hide each other's latency.
#pragma once
#include "kernels.h"

namespace ab
{

// Layout in shared memory: 4 pad words per 32, so that the stages (8 words at
// stride 1, 8, 64, 512 per thread) have no bank conflicts and groups of 4
// words stay 16-byte aligned.
__host__ __device__ constexpr u32 rpad(u32 e) { return e + ((e >> 5) << 2); }

// Twiddles of the 2^LN words in shared memory, as Shoup pairs: the level with
// 2^t polynomials at w[2^t + j]; -w^-1 of the inverse levels at wi[2^t + j], or
// mirrored, w[2^t + 2^t - 1 - j] (domain Q).
struct LevelTw
{
	const uint2 * w, * wi;
	bool mirror;
};

// CNT adjacent pairs from p (aligned to them)
template <int CNT>
__device__ __forceinline__ void load_pairs(const uint2 * p, uint2 (&v)[CNT])
{
	if constexpr (CNT == 1) v[0] = *p;
	else
	{
#pragma unroll
		for (int i = 0; i < CNT / 2; ++i)
		{
			const uint4 q = reinterpret_cast<const uint4 *>(p)[i];
			v[2 * i] = make_uint2(q.x, q.y); v[2 * i + 1] = make_uint2(q.z, q.w);
		}
	}
}

// The twiddles j = x .. x + CNT - 1 of level t (CNT divides x).
template <int CNT, bool INV>
__device__ __forceinline__ void level_tw(const LevelTw & tw, int t, u32 x, uint2 (&v)[CNT])
{
	if (!INV) load_pairs<CNT>(tw.w + (1u << t) + x, v);
	else if (!tw.mirror) load_pairs<CNT>(tw.wi + (1u << t) + x, v);
	else
	{
		uint2 r[CNT];
		load_pairs<CNT>(tw.w + (2u << t) - x - CNT, r);
#pragma unroll
		for (int i = 0; i < CNT; ++i) v[i] = r[CNT - 1 - i];
	}
}

// One level of a group's 2^S words: on group bit s, level t = LN - 1 - (B + s).
template <int LN, int S, int B, bool INV, int SB>
__device__ __forceinline__ void level(u32 (&v)[1 << S], const LevelTw & tw, u32 ohi, u32 p, u32 p2)
{
	constexpr int CNT = 1 << (S - 1 - SB);
	uint2 wv[CNT];
	level_tw<CNT, INV>(tw, LN - 1 - (B + SB), ohi << (S - 1 - SB), wv);
#pragma unroll
	for (int jh = 0; jh < CNT; ++jh)
#pragma unroll
		for (int gl = 0; gl < (1 << SB); ++gl)
		{
			const int g = (jh << (SB + 1)) + gl;
			if (INV) inv_bf(v[g], v[g + (1 << SB)], wv[jh].x, wv[jh].y, p, p2);
			else fwd_bf(v[g], v[g + (1 << SB)], wv[jh].x, wv[jh].y, p, p2);
		}
}

// Levels on index bits B..B+S-1 of the words at src into dst: forward from the
// top one, inverse from the bottom one.
template <int LN, int S, int B, bool INV>
__device__ __forceinline__ void level_stage(const u32 * src, u32 * dst, const LevelTw & tw, u32 tid, u32 NT, u32 p, u32 p2)
{
	constexpr u32 N = 1u << LN;
	for (u32 o = tid; o < (N >> S); o += NT)
	{
		u32 v[1 << S];
		const u32 ohi = o >> B;
		const u32 a0 = rpad((o & ((1u << B) - 1)) | (ohi << (B + S)));
#pragma unroll
		for (int g = 0; g < (1 << S); ++g) v[g] = src[a0 + rpad((u32)g << B)];
		if constexpr (INV)
		{
			level<LN, S, B, true, 0>(v, tw, ohi, p, p2);
			if constexpr (S > 1) level<LN, S, B, true, 1>(v, tw, ohi, p, p2);
			if constexpr (S > 2) level<LN, S, B, true, 2>(v, tw, ohi, p, p2);
		}
		else
		{
			if constexpr (S > 2) level<LN, S, B, false, 2>(v, tw, ohi, p, p2);
			if constexpr (S > 1) level<LN, S, B, false, 1>(v, tw, ohi, p, p2);
			level<LN, S, B, false, 0>(v, tw, ohi, p, p2);
		}
#pragma unroll
		for (int g = 0; g < (1 << S); ++g) dst[a0 + rpad((u32)g << B)] = v[g];
	}
}

// Pointwise product of 4 adjacent degree-1 polynomials (v[2m], v[2m+1]) mod
// (x^2 -+ c), words in [0, 2p); c0 for the first two, c1 for the others (even
// polynomials -c, odd ones +c).  y: the other factor (mul), else a square.
__device__ __forceinline__ void pointwise4(u32 (&v)[8], const u32 (&y)[8], bool mul, uint2 c0, uint2 c1, u32 p, u32 p2, u32 pinv)
{
#pragma unroll
	for (int m = 0; m < 4; ++m)
	{
		const u32 cm = mont_twiddle((m < 2) ? c0 : c1, p);
		poly_product(v[2 * m], v[2 * m + 1], mul ? y[2 * m] : v[2 * m], mul ? y[2 * m + 1] : v[2 * m + 1], mul,
			((m & 1) == 0) ? cm : p - cm, p, p2, pinv);
	}
}

enum BottomMode { BOTTOM_SQUARE = 0, BOTTOM_MUL = 1, BOTTOM_FORWARD = 2 };

// The bottom of a transform, 8 adjacent words per thread: the last two forward
// levels, the pointwise product, the first two inverse levels, in place; or
// (BOTTOM_FORWARD) the last two levels only, the words in [0, 2p) to out.
// op(o, a, b) gives the other factor's words 8 o .. 8 o + 7, out(o, a, b) takes
// the image.
template <int LN, typename Op, typename Out>
__device__ __forceinline__ void level_bottom(u32 * x, int mode, const LevelTw & tw, u32 tid, u32 NT, u32 p, u32 p2, u32 pinv, Op op, Out out)
{
	constexpr u32 N = 1u << LN;
	for (u32 o = tid; o < N / 8; o += NT)
	{
		u32 v[8], y[8];
		uint4 * const xp = reinterpret_cast<uint4 *>(x + rpad(8 * o));
		uint4 a = make_uint4(0, 0, 0, 0), b = a;
		if (mode == BOTTOM_MUL) op(o, a, b);
		y[0] = a.x; y[1] = a.y; y[2] = a.z; y[3] = a.w; y[4] = b.x; y[5] = b.y; y[6] = b.z; y[7] = b.w;
		a = xp[0]; b = xp[1];
		v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
		uint2 w0[1], w1[2];
		level_tw<1, false>(tw, LN - 3, o, w0);
		level_tw<2, false>(tw, LN - 2, 2 * o, w1);
#pragma unroll
		for (int i = 0; i < 4; ++i) fwd_bf(v[i], v[i + 4], w0[0].x, w0[0].y, p, p2);
#pragma unroll
		for (int i = 0; i < 2; ++i)
		{
			fwd_bf(v[i], v[i + 2], w1[0].x, w1[0].y, p, p2);
			fwd_bf(v[i + 4], v[i + 6], w1[1].x, w1[1].y, p, p2);
		}
#pragma unroll
		for (int i = 0; i < 8; ++i) v[i] = red2(v[i], p2);
		if (mode == BOTTOM_FORWARD)
		{
			out(o, make_uint4(v[0], v[1], v[2], v[3]), make_uint4(v[4], v[5], v[6], v[7]));
			continue;
		}
		pointwise4(v, y, mode == BOTTOM_MUL, w1[0], w1[1], p, p2, pinv);
		level_tw<2, true>(tw, LN - 2, 2 * o, w1);
		level_tw<1, true>(tw, LN - 3, o, w0);
#pragma unroll
		for (int i = 0; i < 2; ++i)
		{
			inv_bf(v[i], v[i + 2], w1[0].x, w1[0].y, p, p2);
			inv_bf(v[i + 4], v[i + 6], w1[1].x, w1[1].y, p, p2);
		}
#pragma unroll
		for (int i = 0; i < 4; ++i) inv_bf(v[i], v[i + 4], w0[0].x, w0[0].y, p, p2);
		xp[0] = make_uint4(v[0], v[1], v[2], v[3]);
		xp[1] = make_uint4(v[4], v[5], v[6], v[7]);
	}
}

// A whole transform step: the words at src through all forward levels, the
// pointwise product and all inverse levels into x.  The caller's barrier makes
// src and the tables visible; on return the words of x are written but not yet
// ordered for other threads.
template <int LN, typename Op, typename Out>
__device__ __forceinline__ void level_transform(const u32 * src, u32 * x, int mode, const LevelTw & tw, u32 tid, u32 NT,
	u32 p, u32 pinv, Op op, Out out)
{
	const u32 p2 = 2 * p;
	constexpr int REM = (LN - 3) % 3;
	constexpr int TOP = (REM == 0) ? 3 : REM, BT = LN - TOP;    // the top stage: bits BT..LN-1
	static_assert(LN >= 6 && LN <= 12, "stages above bit 9 are the top one");
	level_stage<LN, TOP, BT, false>(src, x, tw, tid, NT, p, p2);
	__syncthreads();
	if constexpr (BT >= 9) { level_stage<LN, 3, 6, false>(x, x, tw, tid, NT, p, p2); __syncthreads(); }
	if constexpr (BT >= 6) { level_stage<LN, 3, 3, false>(x, x, tw, tid, NT, p, p2); __syncthreads(); }
	level_bottom<LN>(x, mode, tw, tid, NT, p, p2, pinv, op, out);
	if (mode == BOTTOM_FORWARD) return;
	__syncthreads();
	if constexpr (BT >= 6) { level_stage<LN, 3, 3, true>(x, x, tw, tid, NT, p, p2); __syncthreads(); }
	if constexpr (BT >= 9) { level_stage<LN, 3, 6, true>(x, x, tw, tid, NT, p, p2); __syncthreads(); }
	level_stage<LN, TOP, BT, true>(x, x, tw, tid, NT, p, p2);
}

} // namespace ab
