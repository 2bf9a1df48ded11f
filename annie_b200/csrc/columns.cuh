// The column pass: kernel and launch, one translation unit per class
// (columns2.cu .. columns5.cu), and the body for the mixed-size kernel
// (kernels.cu).
#pragma once
#include <type_traits>

#include "kernels.h"
#include "carry.cuh"
#include "launch.cuh"
#include "pdl.cuh"

namespace ab
{

// ================================================================ column pass
// A CTA's tile is CW = 32 columns wide, one lane per column: E predecessor
// columns, whose groups only give the carry into the CTA's first group, then
// the CTA's own columns.  CTA 0 has E = 8 (the mod R / mod Q decision needs
// the final value of the register's last coefficient, whose own predecessor
// group is the 4 columns before it) and 24 own columns, the others E = 4 and
// up to 28; a row of 32 columns is a single CTA without predecessors.  So every
// butterfly task is a full warp of 32 adjacent columns, and a tile row is
// 128 bytes of shared memory without padding.
constexpr int CW = 32;
__host__ __device__ constexpr u32 col_ctas(u32 RC) { return (RC <= 32) ? 1u : 1u + (RC - 24u + 27u) / 28u; }

// Threads of a column-pass CTA: the carry phases have 8 groups of 4 columns
// per row, the butterfly stages KP / 8 times 32 tasks per row, so the thread
// count follows the number of rows.
constexpr int COL_ROW_THREADS = 8, COL_SM_THREADS = 1024;   // per row; per SM (64 registers each)
constexpr int COL_THREADS = 384;                       // fused kernels: every split in one launch
template <int LOG_H, bool WIDE>
struct ColCfg
{
	static constexpr int NT = WIDE ? 32 << LOG_H : ((COL_ROW_THREADS << LOG_H) < 64) ? 64 : (COL_ROW_THREADS << LOG_H);
	static constexpr int MINB = (COL_SM_THREADS / NT < 16) ? COL_SM_THREADS / NT : 16;
};

// One radix-2^S step of the column transform (levels on row bits b..b+S-1)
// for one column of one prime: the 2^S rows that differ in those bits, read
// from src and written to dst (tile or global, row strides ss and ds).
// Global level l (2^l polynomials) works on row bit LOG_H-1-l with twiddle
// tw[2^l + j], j = row >> (LOG_H - l) (forward: w; inverse: -w^-1).
template <int S, bool INV>
__device__ __forceinline__ void col_step(const u32 * src, u32 ss, u32 * dst, u32 ds, int LOG_H, int b, u32 o,
	const uint2 * __restrict__ tw, u32 p, u32 p2)
{
	u32 v[1 << S];
	const u32 row0 = (o & ((1u << b) - 1)) | ((o >> b) << (b + S));
	const u32 * const sp = src + row0 * ss;
#pragma unroll
	for (int g = 0; g < (1 << S); ++g) v[g] = sp[((u32)g << b) * ss];
	const u32 ohi = o >> b;
#pragma unroll
	for (int t = 0; t < S; ++t)
	{
		const int s = INV ? t : (S - 1 - t);
		const int lvl = LOG_H - 1 - (b + s);
		const uint2 * __restrict__ twl = tw + ((1u << lvl) + (ohi << (S - 1 - s)));
#pragma unroll
		for (int jh = 0; jh < (1 << (S - 1 - s)); ++jh)
		{
			const uint2 wv = twl[jh];
#pragma unroll
			for (int gl = 0; gl < (1 << s); ++gl)
			{
				const int g = (jh << (s + 1)) + gl;
				if (INV) inv_bf(v[g], v[g + (1 << s)], wv.x, wv.y, p, p2);
				else fwd_bf(v[g], v[g + (1 << s)], wv.x, wv.y, p, p2);
			}
		}
	}
	u32 * const dp = dst + row0 * ds;
#pragma unroll
	for (int g = 0; g < (1 << S); ++g) dp[((u32)g << b) * ds] = v[g];
}

// The LOG_H column levels in at most two stages: the bottom SB row bits and
// the other ST ones.
template <int LOG_H>
struct ColStages
{
	static constexpr int ST = (LOG_H > 3) ? LOG_H / 2 : 0, SB = LOG_H - ST;
};

// Inverse levels of every tile column, from global memory (x: plane 0, row 0)
// into the tile.
template <int LOG_H, int KP, int NT>
__device__ __forceinline__ void col_inverse(const u32 * __restrict__ x, u32 n, u32 R, u32 gc, bool live, u32 * tile, const uint2 * twk, const TConst & c)
{
	constexpr int SB = ColStages<LOG_H>::SB, ST = ColStages<LOG_H>::ST, PS = CW << LOG_H;
	const int tid = (int)threadIdx.x, u = tid & 31;
	for (int task = tid; task < (KP << (LOG_H - SB + 5)); task += NT)
	{
		const int o = (task >> 5) & ((1 << (LOG_H - SB)) - 1), k = task >> (LOG_H - SB + 5);
		const u32 p = c.p[k];
		if (live) col_step<SB, true>(x + (size_t)k * n + gc, R, tile + k * PS + u, CW, LOG_H, 0, (u32)o, twk + (k << LOG_H), p, 2 * p);
	}
	__syncthreads();
	if constexpr (ST > 0)
	{
		for (int task = tid; task < (KP << (LOG_H - ST + 5)); task += NT)
		{
			const int o = (task >> 5) & ((1 << (LOG_H - ST)) - 1), k = task >> (LOG_H - ST + 5);
			const u32 p = c.p[k];
			col_step<ST, true>(tile + k * PS + u, CW, tile + k * PS + u, CW, LOG_H, SB, (u32)o, twk + (k << LOG_H), p, 2 * p);
		}
		__syncthreads();
	}
}

// Forward levels of the own columns, from the tile into global memory.
template <int LOG_H, int KP, int NT>
__device__ __forceinline__ void col_forward(u32 * tile, u32 * __restrict__ x, u32 n, u32 R, u32 gc, bool own, const uint2 * twk, const TConst & c)
{
	constexpr int SB = ColStages<LOG_H>::SB, ST = ColStages<LOG_H>::ST, PS = CW << LOG_H;
	const int tid = (int)threadIdx.x, u = tid & 31;
	if constexpr (ST > 0)
	{
		for (int task = tid; task < (KP << (LOG_H - ST + 5)); task += NT)
		{
			const int o = (task >> 5) & ((1 << (LOG_H - ST)) - 1), k = task >> (LOG_H - ST + 5);
			const u32 p = c.p[k];
			col_step<ST, false>(tile + k * PS + u, CW, tile + k * PS + u, CW, LOG_H, SB, (u32)o, twk + (k << LOG_H), p, 2 * p);
		}
		__syncthreads();
	}
	for (int task = tid; task < (KP << (LOG_H - SB + 5)); task += NT)
	{
		const int o = (task >> 5) & ((1 << (LOG_H - SB)) - 1), k = task >> (LOG_H - SB + 5);
		const u32 p = c.p[k];
		if (own) col_step<SB, false>(tile + k * PS + u, CW, x + (size_t)k * n + gc, R, LOG_H, 0, (u32)o, twk + (k << LOG_H), p, 2 * p);
	}
}

// Adds d to an exact value (three limbs).
__device__ __forceinline__ void exact_add(u32 (&x)[AB_NW], __int128 d)
{
	const unsigned __int128 v = ((unsigned __int128)x[0] | ((unsigned __int128)x[1] << 32) | ((unsigned __int128)x[2] << 64)) +
	                            (unsigned __int128)d;
	x[0] = (u32)v; x[1] = (u32)(v >> 32); x[2] = (u32)(v >> 64);
}

// Second carry phase for one group of 4 coefficients (kernel.cl:1582-1613):
// f = carry-in, d = the group's unsigned W-bit digits.  The first three become
// balanced, v in [-2^(W-1), 2^(W-1)) with the carry (f + d + 2^(W-1)) >> W;
// the last one absorbs the rest.  x: exact values (three limbs each); the sums
// past the first have CarryLimbs limbs.
template <bool FULL, int L, int PCK>
__device__ __forceinline__ void carry_phase2(const Width & w, const Big<AB_NW> & half, const Big<L> & f, const u32 (&d)[4][DigitLimbs<PCK>::N],
	u32 (&x)[4][AB_NW])
{
	constexpr int ND = DigitLimbs<PCK>::N, CL = CarryLimbs<FULL, L>::N;
	u32 hd[ND];
#pragma unroll
	for (int i = 0; i < ND; ++i) hd[i] = half.l[i];
	Big<CL> g;
	auto balanced = [&](const u32 (&e)[ND], u32 (&v)[AB_NW]) {
		Big<AB_NW> a;
#pragma unroll
		for (int i = 0; i < AB_NW; ++i) a.l[i] = (i < ND) ? e[i % ND] : 0u;
		a = big_sub<AB_NW>(a, half);
#pragma unroll
		for (int i = 0; i < AB_NW; ++i) v[i] = a.l[i];
	};
	{
		Big<L> t = add_digit<L, ND>(add_digit<L, ND>(f, d[0]), hd);
		u32 e[ND];
		split_digit<FULL, L, ND>(t, w, e);
		balanced(e, x[0]);
		g = carry_extend<CL, L>(t);
	}
#pragma unroll
	for (int j = 1; j < 3; ++j)
	{
		g = add_digit<CL, ND>(add_digit<CL, ND>(g, d[j]), hd);
		u32 e[ND];
		split_digit<FULL, CL, ND>(g, w, e);
		balanced(e, x[j]);
	}
	g = add_digit<CL, ND>(g, d[3]);
#pragma unroll
	for (int i = 0; i < AB_NW; ++i) x[3][i] = g.l[i];
}

// The column pass of column group b of nb of candidate cand, by the NT threads
// of the CTA (a multiple of 32); sm: colpass_smem bytes of shared memory.
//
// Bound by the integer multiplier (butterflies 4 units each, CRT about 75 and
// encoding 54 units per coefficient of 6 primes) when the grid fills the GPU,
// by the chain of phases when it does not.  So a coefficient is handled as one
// digit of W = pck lbase bits instead of pck digits (no 128-bit shifts by a
// runtime amount), the residues are the CRT coordinates themselves (crt), the
// exact values go from the carry to their residues in registers, and the first
// and last butterfly stages read and write global memory directly.  B200, one
// domain out, 33.2M bits: 37.6 -> 24.5 us (17.5 M -> 12.1 M warp instructions,
// multiplier floor 8.6 us); a batch of 16 x 1.1M bits 164.8 -> 85.0 us per step.
//
// WIDE: a thread per tile word (32 H threads) and the carry by 4 lanes per
// group (carry.cuh), for launches that do not fill the GPU.  SPARSE: the source
// is SRC_SPARSE (both jobs of the launch).
template <int LOG_H, int K, int PCK, bool WIDE, bool SPARSE, int NT>
__device__ __forceinline__ void colpass_body(ColJob J, const TConst & c, u32 cand, int b, int nb, u32 * sm, int & decision)
{
	constexpr int KP = K + 1, L = K;             // transform primes, limbs of the carry
	constexpr int H = 1 << LOG_H;
	constexpr int PS = H * CW;                   // tile plane stride
	constexpr int ND = DigitLimbs<PCK>::N;
	u32 * const tile = sm;                       // [KP][H][CW]
	u32 * const cw = tile + KP * PS;             // [H][8][L] carry-out words
	u32 * const edge = cw + H * 8 * L;           // [2][4][AB_NW]: the groups that the mod R / mod Q step adjusts
	uint2 * const twc = reinterpret_cast<uint2 *>(edge + 24);   // [3][KP][H] column twiddles

	const u32 amul = (J.mult != nullptr) ? J.mult[cand] : J.a;
	if (amul == 0u) return;                       // inactive batch slot
	{
		const size_t on = (size_t)cand * J.stride_norm, ot = (size_t)cand * J.stride_ntt;
		J.in += (!SPARSE && J.transformed == SRC_NTT) ? ot : on;
		if (J.sub) J.sub += on;
		if (J.out_norm) J.out_norm += on;
		if (J.out_fwd[0]) J.out_fwd[0] += ot;
		if (J.out_fwd[1]) J.out_fwd[1] += ot;
		if (J.out_snap) J.out_snap = (J.snap_flag[cand] != 0u) ? J.out_snap + on : nullptr;
	}
	const int wbits = PCK * ((J.cand != nullptr) ? J.cand[cand].lbase : c.lbase);
	const u32 R = c.R, n = c.n;
	const bool single = (nb == 1);
	const int E = single ? 0 : (b == 0) ? 8 : 4;
	const u32 c0 = (b == 0) ? 0u : 28u * (u32)b - 4u;                  // first own column
	const int WU = min(CW, E + (int)(R - c0)), ng = WU / 4;            // live columns and groups of a row
	const int tid = (int)threadIdx.x;
	// global column of tile column u (CTA 0's predecessors end the previous row)
	auto gcol = [&](int u) -> u32 { return c0 + (u32)(u - E) + ((b == 0 && u < E) ? R : 0u); };
	const int lane = tid & 31;

	// ---- the column twiddles (constant tables)
	for (int idx = tid; idx < KP * H; idx += NT)
	{
		const int k = idx / H, i = idx % H;
		if (i == 0) continue;
		if (!SPARSE && J.transformed == SRC_NTT) twc[idx] = J.wi_in[k * COLTW + i];
		if (J.out_fwd[0] != nullptr) twc[KP * H + idx] = J.w_out[0][k * COLTW + i];
		if (J.out_fwd[1] != nullptr) twc[2 * KP * H + idx] = J.w_out[1][k * COLTW + i];
	}
	if (tid == 0) decision = 0;
	__syncthreads();
	griddep_wait();

	// a group's exact values: normal form out, residues into the tile
	const bool fwd = (J.out_fwd[0] != nullptr) || (J.out_fwd[1] != nullptr);
	auto encode = [&](int row, int u4, const u32 (&x)[4][AB_NW]) {
#pragma unroll
		for (int k = 0; k < KP; ++k)
		{
			u32 r[4];
#pragma unroll
			for (int j = 0; j < 4; ++j) r[j] = encode_res(c, k, x[j][0], x[j][1], x[j][2]);
			*reinterpret_cast<uint4 *>(tile + k * PS + row * CW + 4 * u4) = make_uint4(r[0], r[1], r[2], r[3]);
		}
	};
	// the same for the thread's own word of a WIDE tile
	auto encode1 = [&](const u32 (&x)[AB_NW]) {
#pragma unroll
		for (int k = 0; k < KP; ++k) tile[k * PS + tid] = encode_res(c, k, x[0], x[1], x[2]);
	};
	auto finalize = [&](int row, int u4, const u32 (&x)[4][AB_NW]) {
		const size_t o = (size_t)row * R + gcol(4 * u4);
#pragma unroll
		for (int l = 0; l < AB_NW; ++l)
		{
			const uint4 val = make_uint4(x[0][l], x[1][l], x[2][l], x[3][l]);
			if (J.out_norm) *reinterpret_cast<uint4 *>(J.out_norm + (size_t)l * n + o) = val;
			if (J.out_snap) *reinterpret_cast<uint4 *>(J.out_snap + (size_t)l * n + o) = val;
		}
		if (fwd) encode(row, u4, x);
	};
	auto load_norm = [&](const u32 * src, int row, int u4, u32 (&x)[4][AB_NW]) {
#pragma unroll
		for (int l = 0; l < AB_NW; ++l)
		{
			const uint4 t = *reinterpret_cast<const uint4 *>(src + (size_t)l * n + (size_t)row * R + gcol(4 * u4));
			x[0][l] = t.x; x[1][l] = t.y; x[2][l] = t.z; x[3][l] = t.w;
		}
	};

	if (SPARSE || J.transformed == SRC_NTT)
	{
		// ---- inverse column levels
		auto get_m = [&](u32 i, u32 & d0, u32 & d1, u32 & d2) { d0 = J.in[i]; d1 = J.in[n + i]; d2 = J.in[2 * (size_t)n + i]; };
		if constexpr (!SPARSE) col_inverse<LOG_H, KP, NT>(J.in, n, R, gcol(lane), lane < WU, tile, twc, c);

		const Width w = make_width(wbits);
		const bool full = (w.ws == ND - 1);
		const bool adjust = (J.lower != LOWER_NONE);
		const bool edges = adjust && (b == 0 || b == nb - 1);
		if constexpr (WIDE)
		{
			// a thread per tile word: row tid / 32, column lane
			const int row = tid >> 5, u4 = lane >> 2;
			const u32 j = (u32)lane & 3u;
			const size_t o = (size_t)row * R + gcol(lane);
			Big<L> f = big_zero<L>();
			if (lane < WU)
			{
				u32 sv[AB_NW] = {};
				if (J.sub != nullptr)
				{
#pragma unroll
					for (int l = 0; l < AB_NW; ++l) sv[l] = J.sub[(size_t)l * n + o];
				}
				if constexpr (SPARSE) f = sparse_product<L>(J.cand[cand].sp, (u32)o, n, get_m);
				else
				{
					u32 y[KP];
#pragma unroll
					for (int k = 0; k < KP; ++k) y[k] = tile[k * PS + tid];
					f = crt<L>(c, y);
				}
				if (amul != 1u) f = big_mul_u32<L>(f, amul);
				if (J.sub != nullptr) f = big_sub<L>(f, big_from_exact<L>(sv[0], sv[1], sv[2]));
			}
			u32 d[ND], x[AB_NW];
			if (full) lane_digits<true, L, ND>(f, w, j, d);
			else lane_digits<false, L, ND>(f, w, j, d);
			if (lane < WU && j == 3)
			{
#pragma unroll
				for (int l = 0; l < L; ++l) cw[(tid >> 2) * L + l] = f.l[l];
			}
			__syncthreads();
			const bool mine = (lane >= E && lane < WU);
			const bool top0 = adjust && E == 8 && row == H - 1 && u4 == 1;
			Big<L> cin = big_zero<L>();
			if (j == 0 && (mine || top0))
			{
				int prow = row, pu4 = u4 - 1;
				bool neg = false;
				if (b == 0 && lane == E)
				{
					// first group of a row: its predecessor ends the previous row
					if (E == 0) pu4 = ng - 1;
					if (row > 0) prow = row - 1;
					else { prow = H - 1; neg = (J.nega != 0); }
				}
#pragma unroll
				for (int l = 0; l < L; ++l) cin.l[l] = cw[(prow * 8 + pu4) * L + l];
				if (neg) cin = big_neg<L>(cin);
			}
			if (full) lane_balance<true, L, ND>(cin, d, w, half_of(wbits), j, x);
			else lane_balance<false, L, ND>(cin, d, w, half_of(wbits), j, x);
			if (edges)
			{
				// mod R (+2) / mod Q on the top and bottom coefficients (kernel.cl:1653-1683);
				// CTA 0 re-derives the last coefficient of the register from its
				// predecessor columns
				const bool last = (b == nb - 1) && row == H - 1 && lane == WU - 1;
				if ((last || (top0 && j == 3)) && reaches_width(x, w)) decision = 1;
				__syncthreads();
				if (last && decision) exact_add(x, -((__int128)1 << wbits));
				if (b == 0 && row == 0 && lane == E)
				{
					int dv = 0;
					if (decision) dv += (J.lower == LOWER_Q) ? -1 : 1;
					if (J.lower == LOWER_R_ADD2) dv += 2;
					exact_add(x, (__int128)dv);
				}
			}
			if (mine)
			{
#pragma unroll
				for (int l = 0; l < AB_NW; ++l)
				{
					if (J.out_norm) J.out_norm[(size_t)l * n + o] = x[l];
					if (J.out_snap) J.out_snap[(size_t)l * n + o] = x[l];
				}
				if (fwd) encode1(x);
			}
		}
		else
		{
			// ---- carry phase 1: per group, exact values (CRT), x a, - sub,
			// unsigned digits + carry-out
			for (int idx = tid; idx < H * 8; idx += NT)
			{
				const int row = idx >> 3, u4 = idx & 7;
				if (u4 >= ng) continue;
				u32 xv[KP][4];
				if constexpr (!SPARSE)
				{
#pragma unroll
					for (int k = 0; k < KP; ++k)
					{
						const uint4 t = *reinterpret_cast<const uint4 *>(tile + k * PS + row * CW + 4 * u4);
						xv[k][0] = t.x; xv[k][1] = t.y; xv[k][2] = t.z; xv[k][3] = t.w;
					}
				}
				u32 sv[4][AB_NW];
				if (J.sub != nullptr) load_norm(J.sub, row, u4, sv);
				Big<L> f = big_zero<L>();
				u32 dg[4][ND];
				auto digits = [&](auto is_full) {
#pragma unroll
					for (int j = 0; j < 4; ++j)
					{
						Big<L> V;
						if constexpr (SPARSE) V = sparse_product<L>(J.cand[cand].sp, (u32)row * R + gcol(4 * u4) + (u32)j, n, get_m);
						else
						{
							u32 rr[KP];
#pragma unroll
							for (int k = 0; k < KP; ++k) rr[k] = xv[k][j];
							V = crt<L>(c, rr);
						}
						if (amul != 1u) V = big_mul_u32<L>(V, amul);
						if (J.sub != nullptr) V = big_sub<L>(V, big_from_exact<L>(sv[j][0], sv[j][1], sv[j][2]));
						f = (j == 0) ? V : big_add<L>(f, V);
						split_digit<decltype(is_full)::value, L, ND>(f, w, dg[j]);
					}
				};
				if (full) digits(std::true_type{});
				else digits(std::false_type{});
#pragma unroll
				for (int l = 0; l < ND; ++l)
					*reinterpret_cast<uint4 *>(tile + l * PS + row * CW + 4 * u4) = make_uint4(dg[0][l], dg[1][l], dg[2][l], dg[3][l]);
#pragma unroll
				for (int l = 0; l < L; ++l) cw[idx * L + l] = f.l[l];
			}
			__syncthreads();

			// ---- carry phase 2: add the previous group's carry-out, balanced
			// values; then the outputs of the group.  Each thread reads and writes
			// only its own group of the tile.
			const Big<AB_NW> half = half_of(wbits);
			for (int idx = tid; idx < H * 8; idx += NT)
			{
				const int row = idx >> 3, u4 = idx & 7;
				if (u4 >= ng) continue;
				// CTA 0 re-derives the last coefficient of the register from its
				// predecessor columns, for the mod R / mod Q decision
				const bool top0 = adjust && E == 8 && row == H - 1 && u4 == 1;
				if (4 * u4 < E && !top0) continue;
				int prow = row, pu4 = u4 - 1;
				bool neg = false;
				if (b == 0 && 4 * u4 == E)
				{
					// first group of a row: its predecessor ends the previous row
					if (E == 0) pu4 = ng - 1;
					if (row > 0) prow = row - 1;
					else { prow = H - 1; neg = (J.nega != 0); }
				}
				Big<L> f;
#pragma unroll
				for (int l = 0; l < L; ++l) f.l[l] = cw[(prow * 8 + pu4) * L + l];
				if (neg) f = big_neg<L>(f);
				u32 dg[4][ND];
#pragma unroll
				for (int l = 0; l < ND; ++l)
				{
					const uint4 t = *reinterpret_cast<const uint4 *>(tile + l * PS + row * CW + 4 * u4);
					dg[0][l] = t.x; dg[1][l] = t.y; dg[2][l] = t.z; dg[3][l] = t.w;
				}
				u32 ex[4][AB_NW];
				if (full) carry_phase2<true, L, PCK>(w, half, f, dg, ex);
				else carry_phase2<false, L, PCK>(w, half, f, dg, ex);
				const bool first = (b == 0) && row == 0 && 4 * u4 == E;
				const bool last = (b == nb - 1) && row == H - 1 && u4 == ng - 1;
				if (adjust && (first || last || top0))
				{
					if ((last || top0) && reaches_width(ex[3], w)) decision = 1;
					if (!top0)
					{
#pragma unroll
						for (int j = 0; j < 4; ++j)
#pragma unroll
							for (int l = 0; l < AB_NW; ++l) edge[(last ? 12 : 0) + 3 * j + l] = ex[j][l];
					}
				}
				else finalize(row, u4, ex);
			}

			// ---- mod R (+2) / mod Q on the top and bottom coefficients (kernel.cl:1653-1683)
			if (edges)
			{
				__syncthreads();
				if (tid < 2 && ((tid == 0) ? b == 0 : b == nb - 1))
				{
					u32 ex[4][AB_NW];
#pragma unroll
					for (int j = 0; j < 4; ++j)
#pragma unroll
						for (int l = 0; l < AB_NW; ++l) ex[j][l] = edge[12 * tid + 3 * j + l];
					if (tid == 0)
					{
						int d = 0;
						if (decision) d += (J.lower == LOWER_Q) ? -1 : 1;
						if (J.lower == LOWER_R_ADD2) d += 2;
						exact_add(ex[0], (__int128)d);
						finalize(0, E / 4, ex);
					}
					else
					{
						if (decision) exact_add(ex[3], -((__int128)1 << wbits));
						finalize(H - 1, ng - 1, ex);
					}
				}
			}
		}
	}

	// ---- the first LA forward levels of the result in one or two domains: the
	// residues of a transformed source are in the tile; those of a normal-form
	// source, and of the second domain, come from the normal form in global memory
	const bool carried = SPARSE || (J.transformed == SRC_NTT);
	bool in_tile = carried;
	const bool own = (lane >= E && lane < WU);
#pragma unroll 1
	for (int dom = 0; dom < 2; ++dom)
	{
		u32 * const out = (dom == 0) ? J.out_fwd[0] : J.out_fwd[1];
		if (out == nullptr) continue;
		if (!in_tile)
		{
			__syncthreads();
			const u32 * src = carried ? J.out_norm : J.in;
			if constexpr (WIDE)
			{
				if (own)
				{
					const size_t o = (size_t)(tid >> 5) * R + gcol(lane);
					const u32 x[AB_NW] = { src[o], src[(size_t)n + o], src[2 * (size_t)n + o] };
					encode1(x);
				}
			}
			else
			{
				for (int idx = tid; idx < H * 8; idx += NT)
				{
					const int row = idx >> 3, u4 = idx & 7;
					if (4 * u4 < E || u4 >= ng) continue;
					u32 x[4][AB_NW];
					load_norm(src, row, u4, x);
					encode(row, u4, x);
				}
			}
		}
		__syncthreads();
		col_forward<LOG_H, KP, NT>(tile, out, n, R, gcol(lane), own, twc + (1 + dom) * KP * H, c);
		in_tile = false;
	}
}

template <int LOG_H, int K, int PCK, bool WIDE, bool SPARSE>
__global__ void __launch_bounds__(ColCfg<LOG_H, WIDE>::NT, ColCfg<LOG_H, WIDE>::MINB) k_colpass(const ColJobs jobs, const TConst c)
{
	extern __shared__ __align__(16) u32 sm[];
	__shared__ int decision;
	colpass_body<LOG_H, K, PCK, WIDE, SPARSE, ColCfg<LOG_H, WIDE>::NT>((blockIdx.y == 0) ? jobs.j[0] : jobs.j[1], c, blockIdx.z, (int)blockIdx.x, (int)gridDim.x, sm, decision);
}

template <int LOG_H, int K, int PCK, bool WIDE, bool SPARSE>
static cudaError_t colpass_w(const Geometry & g, const TConst & c, const ColJobs & jobs, int njobs, cudaStream_t s, int ncand)
{
	const size_t smem = colpass_smem(g, K + 1);
	static std::atomic<unsigned long long> attr_done{0};
	const cudaError_t e = allow_dynamic_smem(k_colpass<LOG_H, K, PCK, WIDE, SPARSE>, smem, attr_done);
	if (e != cudaSuccess) return e;
	if (ncand == 0) return cudaSuccess;      // set-up only (before a stream capture)
	const dim3 grid(g.NC, (unsigned)njobs, (unsigned)ncand);
	return launch_pdl(k_colpass<LOG_H, K, PCK, WIDE, SPARSE>, grid, dim3(ColCfg<LOG_H, WIDE>::NT), smem, s, jobs, c);
}

template <int LOG_H, int K, int PCK, bool WIDE>
static cudaError_t colpass_s(const Geometry & g, const TConst & c, const ColJobs & jobs, int njobs, cudaStream_t s, int ncand)
{
	if (ncand == 0)
	{
		const cudaError_t e = colpass_w<LOG_H, K, PCK, WIDE, true>(g, c, jobs, njobs, s, 0);
		return (e != cudaSuccess) ? e : colpass_w<LOG_H, K, PCK, WIDE, false>(g, c, jobs, njobs, s, 0);
	}
	return (jobs.j[0].transformed == SRC_SPARSE) ? colpass_w<LOG_H, K, PCK, WIDE, true>(g, c, jobs, njobs, s, ncand)
	                                             : colpass_w<LOG_H, K, PCK, WIDE, false>(g, c, jobs, njobs, s, ncand);
}

// A thread per tile word (WIDE) up to 16 rows and COL_WIDE_CTAS CTAs: where
// the launch leaves SMs idle, the shorter chains win (us per squaring, grouped /
// wide: 524k bits 28.6 / 23.1, 2M bits 34.2 / 31.1, 4M bits 41.7 / 38.4); with
// 32 rows a CTA has 1,024 threads and costs more to start than it saves (6.6M
// bits, 147 CTAs: 52.1 / 60.7).
constexpr u32 COL_WIDE_CTAS = 296;
template <int LOG_H, int K, int PCK>
static cudaError_t colpass_t(const Geometry & g, const TConst & c, const ColJobs & jobs, int njobs, cudaStream_t s, int ncand)
{
	if constexpr (LOG_H <= 4)
	{
		if (ncand == 0)
		{
			const cudaError_t e = colpass_s<LOG_H, K, PCK, true>(g, c, jobs, njobs, s, 0);
			if (e != cudaSuccess) return e;
		}
		else if (g.NC * (u32)njobs * (u32)ncand <= COL_WIDE_CTAS) return colpass_s<LOG_H, K, PCK, true>(g, c, jobs, njobs, s, ncand);
	}
	return colpass_s<LOG_H, K, PCK, false>(g, c, jobs, njobs, s, ncand);
}

template <int K, int PCK>
static cudaError_t colpass_k(const Geometry & g, const TConst & c, const ColJobs & jobs, int njobs, cudaStream_t s, int ncand)
{
	switch (g.LA)
	{
	case 1: return colpass_t<1, K, PCK>(g, c, jobs, njobs, s, ncand);
	case 2: return colpass_t<2, K, PCK>(g, c, jobs, njobs, s, ncand);
	case 3: return colpass_t<3, K, PCK>(g, c, jobs, njobs, s, ncand);
	case 4: return colpass_t<4, K, PCK>(g, c, jobs, njobs, s, ncand);
	case 5: return colpass_t<5, K, PCK>(g, c, jobs, njobs, s, ncand);
	case 6: return colpass_t<6, K, PCK>(g, c, jobs, njobs, s, ncand);
	default: return cudaErrorInvalidValue;
	}
}

} // namespace ab
