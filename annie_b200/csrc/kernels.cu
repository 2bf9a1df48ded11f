// NTT passes of the modular-squaring engine, sm_100a.
//
// Mathematics (reference: ocl/kernel.cl and src/transformGPU.h of galloty/annie):
// per transform prime p_k, a register is n = 2^ln values.  The forward
// transform is LN-1 radix-2 levels; the level with S polynomials maps each
// block of 2m = n/S coefficients mod (x^2m - c^2) to mod (x^m - c) and
// (x^m + c) with c = w[S + j] (j = block index, twiddle table in bit-reversed
// order, transformGPU.h:117-160).  The product of the resulting degree-1
// polynomials is taken mod (x^2 -+ w[n/4 + q/2]) (kernel.cl:230-256), and the
// inverse levels undo the forward ones.  The transform primes are below 2^30,
// so values stay lazily reduced ([0, 4p) forward, [0, 2p) inverse; see
// arith.cuh) and every butterfly is one Shoup product and three adds.  Only
// the exact coefficient values that the carry produces are visible outside,
// and they do not depend on the primes or the order of the butterflies.
//
// The passes split the n coefficients 2-D (row*R + col): the column pass owns
// the first LA levels (all H rows of up to 28 adjacent columns, all KP primes,
// in shared memory) and the row pass owns the last LB levels (one row of one
// prime per CTA, 16 coefficients per thread in registers).
#include <atomic>
#include <type_traits>
#include <utility>

#include "kernels.h"
#include "columns.cuh"
#include "launch.cuh"
#include "pdl.cuh"

namespace ab
{

// ================================================================ row pass
// A CTA transforms one row (R = 2^(LB+1) words) of one prime: levels
// t = 0..LB-1 of the row touch bit LB-t of the in-row index.  Each thread
// holds 16 words; a stage applies S <= 4 levels to groups of 2^S words in
// registers, and stages exchange through shared memory.  The last stage owns
// bits 4..1; bit 0 (the two halves of a degree-1 polynomial) comes from the
// thread index, so the pointwise product pairs lane 2m with lane 2m+1.
// Stage loops are rolled (runtime bit positions) to keep the code small.
//
// Bound by the integer multiplier (about 370 units of one IMAD per coefficient
// of 6 primes, 10.4 us at 33.2M bits) and by latency: half of the pass is its
// last stage, whose lines are touched ahead (rp_touch).  33.2M bits, multiply:
// 33.8 -> 26.6 us.  8 words per thread with the row's twiddles in shared memory
// measured slower (33.2M bits 171 -> 177 us per squaring): more stages, more
// shared-memory traffic.
constexpr int RP_EPT = 16;

// Twiddles of the row pass: the forward levels read w; the inverse levels
// read the -w^-1 table wi (domain R) or, for domain Q (wi == null), the
// forward table at the mirrored position of the level: the level with s
// polynomials holds indices [s, 2s), and index i mirrors to 3s - 1 - i.
struct RowTw
{
	const uint2 * w;
	const uint2 * wi;
	u32 H;
};

template <int S, bool INV, int MIR>
__device__ __forceinline__ void rp_radix(u32 (&v)[RP_EPT], u32 tid, u32 T, int b, int LB, const RowTw & tw,
	u32 Hr, u32 p, u32 p2)
{
	constexpr int G = RP_EPT >> S;
#pragma unroll
	for (int x = 0; x < G; ++x)
	{
		const u32 ohi = (tid + T * (u32)x) >> b;
#pragma unroll
		for (int ss = 0; ss < S; ++ss)
		{
			const int s = INV ? ss : (S - 1 - ss);
			const int t = LB - b - s;
			const u32 i0 = (Hr << t) + (ohi << (S - 1 - s));
			// CNT = 2^(S-1-s) adjacent pairs, aligned to them: 16-byte loads
			uint2 wv[1 << (S - 1)];
			const int CNT = 1 << (S - 1 - s);
			const bool mirror = INV && (MIR < 0 ? tw.wi == nullptr : MIR != 0);
			const uint2 * const wp = !INV ? tw.w + i0 : !mirror ? tw.wi + i0 : tw.w + (3u * (tw.H << t) - i0 - (u32)CNT);
			if (CNT == 1) wv[0] = __ldg(wp);
			else
			{
#pragma unroll
				for (int i = 0; i < CNT / 2; ++i)
				{
					const uint4 q = __ldg(reinterpret_cast<const uint4 *>(wp) + i);
					wv[2 * i] = make_uint2(q.x, q.y); wv[2 * i + 1] = make_uint2(q.z, q.w);
				}
				if (mirror)
				{
#pragma unroll
					for (int i = 0; i < CNT / 2; ++i) { const uint2 q = wv[i]; wv[i] = wv[CNT - 1 - i]; wv[CNT - 1 - i] = q; }
				}
			}
#pragma unroll
			for (int jh = 0; jh < (1 << (S - 1 - s)); ++jh)
			{
#pragma unroll
				for (int gl = 0; gl < (1 << s); ++gl)
				{
					const int g = x * (1 << S) + (jh << (s + 1)) + gl;
					if (INV) inv_bf(v[g], v[g + (1 << s)], wv[jh].x, wv[jh].y, p, p2);
					else fwd_bf(v[g], v[g + (1 << s)], wv[jh].x, wv[jh].y, p, p2);
				}
			}
		}
	}
}

// Stage addressing: the 2^S words of a group are e0 + g 2^b.  In the padded
// shared layout they are pad(e0) + g D with D = 2^b + 2^(b-4) for b >= 5, and
// D = 2 for the last stage (b = 1, the group stays inside one 32-word block).
__device__ __forceinline__ u32 rp_pad(u32 e) { return e + ((e >> 5) << 1); }

__device__ __forceinline__ u32 rp_base(u32 tid, u32 T, int x, int S, int b)
{
	const u32 o = tid + T * (u32)x;
	return (o & ((1u << b) - 1)) | ((o >> b) << (b + S));
}
__device__ __forceinline__ u32 rp_step(int b) { return (b >= 5) ? (1u << b) + (1u << (b - 4)) : (1u << b); }

template <int S>
__device__ __forceinline__ void rp_load_smem(u32 (&v)[RP_EPT], const u32 * sm, u32 tid, u32 T, int b)
{
	const u32 D = rp_step(b);
#pragma unroll
	for (int x = 0; x < (RP_EPT >> S); ++x)
	{
		const u32 * a = sm + rp_pad(rp_base(tid, T, x, S, b));
#pragma unroll
		for (int g = 0; g < (1 << S); ++g) v[x * (1 << S) + g] = a[g * D];
	}
}

template <int S>
__device__ __forceinline__ void rp_store_smem(const u32 (&v)[RP_EPT], u32 * sm, u32 tid, u32 T, int b)
{
	const u32 D = rp_step(b);
#pragma unroll
	for (int x = 0; x < (RP_EPT >> S); ++x)
	{
		u32 * a = sm + rp_pad(rp_base(tid, T, x, S, b));
#pragma unroll
		for (int g = 0; g < (1 << S); ++g) a[g * D] = v[x * (1 << S) + g];
	}
}

template <int S>
__device__ __forceinline__ void rp_load_global(u32 (&v)[RP_EPT], const u32 * __restrict__ x, u32 tid, u32 T, int b)
{
#pragma unroll
	for (int xx = 0; xx < (RP_EPT >> S); ++xx)
	{
		const u32 * a = x + rp_base(tid, T, xx, S, b);
#pragma unroll
		for (int g = 0; g < (1 << S); ++g) v[xx * (1 << S) + g] = a[(u32)g << b];
	}
}

template <int S>
__device__ __forceinline__ void rp_store_global(const u32 (&v)[RP_EPT], u32 * __restrict__ x, u32 tid, u32 T, int b)
{
#pragma unroll
	for (int xx = 0; xx < (RP_EPT >> S); ++xx)
	{
		u32 * a = x + rp_base(tid, T, xx, S, b);
#pragma unroll
		for (int g = 0; g < (1 << S); ++g) a[(u32)g << b] = v[xx * (1 << S) + g];
	}
}

// Pointwise product of the degree-1 polynomials (x0, x1) mod (x^2 -+ c):
// lane 2m holds the x0 of the thread pair's 16 polynomials, lane 2m+1 the x1.
// Each lane computes 8 whole products (even lane: slots 0..7, odd: 8..15).
// Inputs: [0, 4p) from the forward levels, the other operand in [0, 2p);
// a factor 2^-32, which the image factors remove (crt); outputs in [0, 2p) for
// the inverse levels.
// w1: the 8 twiddles of the thread pair's last forward level (just read by
// the forward stage, so an L1 hit), which are the polynomials' c.
__device__ __forceinline__ void rp_pointwise(u32 (&v)[RP_EPT], const u32 * __restrict__ xp, const bool is_mul, u32 tid, u32 NT,
	const uint2 * __restrict__ w1, u32 p, u32 p2, u32 pinv)
{
	// tid: virtual thread (its 16 words are the last-stage elements
	// 32*(tid>>1) + (tid&1) + 2g); NT: physical threads of the CTA (warp mask)
	const bool odd = (tid & 1) != 0;
	const unsigned mask = (NT >= 32) ? 0xffffffffu : ((1u << NT) - 1);
	// the other factor's words of the lane's 8 polynomials are adjacent
	const uint4 * const xq = reinterpret_cast<const uint4 *>(xp) + (tid << 2);
	uint4 op = make_uint4(0, 0, 0, 0);
#pragma unroll
	for (int i = 0; i < 8; ++i)
	{
		if (is_mul && (i & 1) == 0) op = __ldg(xq + (i >> 1));
		const u32 r = __shfl_xor_sync(mask, odd ? v[i] : v[8 + i], 1);
		const u32 x0 = red2(odd ? r : v[i], p2), x1 = red2(odd ? v[8 + i] : r, p2);
		const int slot = odd ? 8 + i : i;   // polynomial slot; parity = sign
		const uint2 cwp = __ldg(w1 + (odd ? 4 + (i >> 1) : (i >> 1)));
		const u32 cm = mont_twiddle(cwp, p);
		u32 y0 = x0, y1 = x1;
		poly_product(y0, y1, !is_mul ? x0 : ((i & 1) == 0) ? op.x : op.z, !is_mul ? x1 : ((i & 1) == 0) ? op.y : op.w, is_mul,
			((slot & 1) == 0) ? cm : p - cm, p, p2, pinv);
		const u32 r2 = __shfl_xor_sync(mask, odd ? y0 : y1, 1);
		if (odd) { v[8 + i] = y1; v[i] = r2; }
		else { v[i] = y0; v[8 + i] = r2; }
	}
}

template <int N>
__device__ __forceinline__ void reduce_all(u32 (&v)[N], u32 p2)
{
#pragma unroll
	for (int i = 0; i < N; ++i) v[i] = red2(v[i], p2);
}

// Physical threads of a row-pass CTA: 16 words per virtual thread, at most
// 256 threads, each running R / (16 * threads) rounds per stage.  The kernel
// is compiled for 3 CTAs per SM (80 registers, no spills): the grids of the
// long lengths have 2.6 per SM (33.2M bits: 384), and 4 of them at 64 registers
// measured the same there and slower below (us per squaring, 4 / 3: 33.2M bits
// 150.2 / 150.4, 6.6M bits 51.4 / 48.2, 2M bits 29.9 / 26.9).  128 threads:
// 185.5 at 33.2M bits; 512: 155.5.
constexpr u32 ROW_THREADS = 256;
template <int LOG_R>
struct RowCfg
{
	static constexpr u32 T = (1u << LOG_R) / RP_EPT;             // virtual threads
	static constexpr u32 NT = (T < ROW_THREADS) ? T : ROW_THREADS;   // physical threads
	static constexpr u32 RND = T / NT;
	static constexpr int MINB = 3;
	static constexpr size_t SMEM = sizeof(u32) * ((1u << LOG_R) + (1u << LOG_R) / 16);   // padded row
};

// Starts the load of a line that is read later (to L1; the value is dropped).
__device__ __forceinline__ void touch(const void * p)
{
	u32 v;
	asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(v) : "l"(p));
}

// What the last stage of a row reads from global memory, per warp of virtual
// threads vt0 .. vt0 + 31 (512 words): 15 lines of forward twiddles, 15 of
// inverse ones (levels LB-4 .. LB-1: 128 << i bytes at level LB-4+i), and 16
// of the other factor.  Touched ahead of the barrier before that stage, so
// that its 8 dependent levels find their twiddles in L1.
__device__ __forceinline__ void rp_touch(u32 vt0, u32 lane, int LB, const RowTw & tw, u32 Hr, const u32 * xp)
{
	const u32 j = lane & 15;
	if (j < 15)
	{
		// line j: level i = 0, 1, 2, 3 has lines 2^i - 1 .. 2^(i+1) - 2
		const u32 i = 31u - (u32)__clz((int)(j + 1)), t = (u32)LB - 4u + i;
		const u32 i0 = (Hr << t) + (vt0 << i >> 1) + (((j + 1) - (1u << i)) << 4);   // 16 pairs a line
		touch(lane < 16 ? tw.w + i0 : tw.wi != nullptr ? tw.wi + i0 : tw.w + (3u * (tw.H << t) - 16u - i0));
	}
	if (xp != nullptr && lane < 16) touch(xp + (vt0 << 4) + (lane << 5));
}

// The row pass of row bx (prime k = bx / HR, row r) of candidate cand, by P
// threads (tid < P) sharing the padded row buffer sm.  When P exceeds the
// row's virtual threads T, the threads above T only take part in the
// barriers.  mask_nt: threads of the CTA, for the shuffle masks.
// MODE, MIR: the job's RowMode and whether its inverse twiddles are the
// mirrored forward ones (domain Q), or -1 where only the job knows.
template <int LOG_R, u32 P, int MODE, int MIR>
__device__ __forceinline__ void rowpass_body(const RowJob & J, const TConst & c, u32 cand, u32 bx, u32 tid, u32 * sm, u32 mask_nt)
{
	constexpr int LB = LOG_R - 1;
	constexpr u32 T = RowCfg<LOG_R>::T, NT = P, RND = (T + P - 1) / P;
	constexpr bool IDLE = P > T;                                  // some threads have no virtual thread
	constexpr int NL = LB - 4;                                    // levels above the last stage
	constexpr int S0 = (NL % 4 == 0) ? 4 : NL % 4;                // first stage (when NL > 0)
	constexpr int NS = (NL == 0) ? 0 : 1 + (NL - S0) / 4;        // stages above the last
	constexpr int B0 = LB + 1 - S0;

	const int mode = (MODE < 0) ? J.mode : MODE;
	const size_t cofs = (size_t)cand * J.stride;
	const u32 k = bx / c.HR, r = bx - k * c.HR;
	const u32 p = c.p[k], p2 = 2 * p, pinv = c.pinv[k];
	u32 * __restrict__ x = J.x + cofs + (size_t)k * c.n + (size_t)r * (1u << LOG_R);
	RowTw tw;
	tw.w = J.w + (size_t)k * (c.n >> 1);
	tw.wi = (J.wi != nullptr) ? J.wi + (size_t)k * (c.n >> 1) : nullptr;
	tw.H = c.HR;
	const u32 * __restrict__ xp = (mode == ROW_MUL) ? J.xp + cofs + (size_t)k * c.n + (size_t)r * (1u << LOG_R) : nullptr;
	const u32 Hr = c.HR + r;
	// threads of a shuffle: with idle threads, only the first T of the first warp
	const u32 mnt = (IDLE && T < 32) ? T : mask_nt;
	u32 v[RP_EPT];
	// twiddles of the last forward level of virtual thread vt: the c of its polynomials
	auto w1 = [&](u32 vt) { return tw.w + (Hr << (LB - 1)) + ((vt >> 1) << 3); };
	griddep_wait();

	if constexpr (NS == 0)
	{
#pragma unroll 1
		for (u32 rr = 0; rr < RND; ++rr)
		{
			const u32 vt = tid + rr * NT;
			if (IDLE && vt >= T) continue;
			rp_load_global<4>(v, x, vt, T, 1);
			rp_radix<4, false, MIR>(v, vt, T, 1, LB, tw, Hr, p, p2);
			if (mode != ROW_FWD_ONLY)
			{
				rp_pointwise(v, xp, mode == ROW_MUL, vt, mnt, w1(vt), p, p2, pinv);
				rp_radix<4, true, MIR>(v, vt, T, 1, LB, tw, Hr, p, p2);
			}
			else reduce_all(v, p2);
			rp_store_global<4>(v, x, vt, T, 1);
		}
		return;
	}
	else
	{
		// ---- forward: stage 0 from global, then stages of 4 levels via smem
#pragma unroll 1
		for (u32 rr = 0; rr < RND; ++rr)
		{
			const u32 vt = tid + rr * NT;
			if (IDLE && vt >= T) continue;
			rp_load_global<S0>(v, x, vt, T, B0);
			rp_radix<S0, false, MIR>(v, vt, T, B0, LB, tw, Hr, p, p2);
			rp_store_smem<S0>(v, sm, vt, T, B0);
		}
		int b = B0;
#pragma unroll 1
		for (int i = 1; i < NS; ++i)
		{
			__syncthreads();
			b -= 4;
#pragma unroll 1
			for (u32 rr = 0; rr < RND; ++rr)
			{
				const u32 vt = tid + rr * NT;
				if (IDLE && vt >= T) continue;
				rp_load_smem<4>(v, sm, vt, T, b);
				rp_radix<4, false, MIR>(v, vt, T, b, LB, tw, Hr, p, p2);
				rp_store_smem<4>(v, sm, vt, T, b);
			}
		}
		const bool ahead = (T >= 32) && mode != ROW_FWD_ONLY;
		if (ahead && tid < T) rp_touch(tid & ~31u, tid & 31, LB, tw, Hr, xp);
		__syncthreads();

		// ---- last stage (bits 4..1), pointwise, inverse last stage
#pragma unroll 1
		for (u32 rr = 0; rr < RND; ++rr)
		{
			const u32 vt = tid + rr * NT;
			if (IDLE && vt >= T) continue;
			if (ahead && vt + NT < T) rp_touch((vt + NT) & ~31u, tid & 31, LB, tw, Hr, xp);
			rp_load_smem<4>(v, sm, vt, T, 1);
			rp_radix<4, false, MIR>(v, vt, T, 1, LB, tw, Hr, p, p2);
			if (mode == ROW_FWD_ONLY)
			{
				reduce_all(v, p2);
				rp_store_global<4>(v, x, vt, T, 1);
				continue;
			}
			rp_pointwise(v, xp, mode == ROW_MUL, vt, mnt, w1(vt), p, p2, pinv);
			rp_radix<4, true, MIR>(v, vt, T, 1, LB, tw, Hr, p, p2);
			rp_store_smem<4>(v, sm, vt, T, 1);
		}
		if (mode == ROW_FWD_ONLY) return;

		// ---- inverse: back up through smem, stage 0 to global
		b = 1;
#pragma unroll 1
		for (int i = NS - 1; i >= 1; --i)
		{
			__syncthreads();
			b += 4;
#pragma unroll 1
			for (u32 rr = 0; rr < RND; ++rr)
			{
				const u32 vt = tid + rr * NT;
				if (IDLE && vt >= T) continue;
				rp_load_smem<4>(v, sm, vt, T, b);
				rp_radix<4, true, MIR>(v, vt, T, b, LB, tw, Hr, p, p2);
				rp_store_smem<4>(v, sm, vt, T, b);
			}
		}
		__syncthreads();
#pragma unroll 1
		for (u32 rr = 0; rr < RND; ++rr)
		{
			const u32 vt = tid + rr * NT;
			if (IDLE && vt >= T) continue;
			rp_load_smem<S0>(v, sm, vt, T, B0);
			rp_radix<S0, true, MIR>(v, vt, T, B0, LB, tw, Hr, p, p2);
			rp_store_global<S0>(v, x, vt, T, B0);
		}
	}
}

template <int LOG_R, int MODE>
__global__ void __launch_bounds__(RowCfg<LOG_R>::NT, RowCfg<LOG_R>::MINB) k_rowpass(const RowJobs jobs, const TConst c)
{
	extern __shared__ __align__(16) u32 sm[];
	const RowJob J = (blockIdx.y == 0) ? jobs.j[0] : jobs.j[1];
	const u32 cand = blockIdx.z;
	if (J.active != nullptr && J.active[cand] == 0u) return;
	constexpr u32 NT = RowCfg<LOG_R>::NT;
	if (J.wi != nullptr) rowpass_body<LOG_R, NT, MODE, 0>(J, c, cand, blockIdx.x, threadIdx.x, sm, NT);
	else rowpass_body<LOG_R, NT, MODE, 1>(J, c, cand, blockIdx.x, threadIdx.x, sm, NT);
}

// ================================================================ mixed-size passes
// The class of CTA bid and the CTA's job, candidate and row / column group.
struct FusedCta
{
	int ci;
	u32 job, cand, bx;
};

template <typename Pass>
__device__ __forceinline__ FusedCta fused_cta(const Pass * __restrict__ d, u32 bid)
{
	FusedCta f;
	int ci = 0;
	while (ci + 1 < d->nclass && bid >= d->begin[ci + 1]) ++ci;
	const u32 local = bid - d->begin[ci], nbx = d->nbx[ci];
	const u32 cj = local / nbx;
	f.ci = ci;
	f.bx = local - cj * nbx;
	f.job = cj % d->njobs[ci];
	f.cand = cj / d->njobs[ci];
	return f;
}

// The class's constants into shared memory (they come from a table written
// when the group was set up, so before griddep_wait).
__device__ __forceinline__ void fused_consts(TConst & cs, const TConst * __restrict__ tcs, int ci)
{
	const u32 * src = reinterpret_cast<const u32 *>(tcs + ci);
	u32 * dst = reinterpret_cast<u32 *>(&cs);
	for (u32 i = threadIdx.x; i < sizeof(TConst) / 4; i += blockDim.x) dst[i] = __ldg(src + i);
	__syncthreads();
}

__global__ void __launch_bounds__(AB_FUSED_ROW_THREADS, 4) k_fused_rowpass(const FusedRowPass * __restrict__ d, const TConst * __restrict__ tcs)
{
	extern __shared__ __align__(16) u32 sm[];
	__shared__ TConst cs;
	const FusedCta f = fused_cta(d, blockIdx.x);
	const RowJob J = d->jobs[f.ci].j[f.job];
	if (J.active != nullptr && J.active[f.cand] == 0u) return;
	fused_consts(cs, tcs, f.ci);
	constexpr u32 P = AB_FUSED_ROW_THREADS;
	switch (d->log_r[f.ci])
	{
	case 5: rowpass_body<5, P, -1, -1>(J, cs, f.cand, f.bx, threadIdx.x, sm, P); break;
	case 6: rowpass_body<6, P, -1, -1>(J, cs, f.cand, f.bx, threadIdx.x, sm, P); break;
	case 7: rowpass_body<7, P, -1, -1>(J, cs, f.cand, f.bx, threadIdx.x, sm, P); break;
	case 8: rowpass_body<8, P, -1, -1>(J, cs, f.cand, f.bx, threadIdx.x, sm, P); break;
	case 9: rowpass_body<9, P, -1, -1>(J, cs, f.cand, f.bx, threadIdx.x, sm, P); break;
	case 10: rowpass_body<10, P, -1, -1>(J, cs, f.cand, f.bx, threadIdx.x, sm, P); break;
	case 11: rowpass_body<11, P, -1, -1>(J, cs, f.cand, f.bx, threadIdx.x, sm, P); break;
	case 12: rowpass_body<12, P, -1, -1>(J, cs, f.cand, f.bx, threadIdx.x, sm, P); break;
	case 13: rowpass_body<13, P, -1, -1>(J, cs, f.cand, f.bx, threadIdx.x, sm, P); break;
	case 14: rowpass_body<14, P, -1, -1>(J, cs, f.cand, f.bx, threadIdx.x, sm, P); break;
	default: break;
	}
}

#define AB_FUSED_COL(LH, KK, PP) \
	case LH * 8 + KK: colpass_body<LH, KK, PP, false, false, COL_THREADS>(J, cs, f.cand, (int)f.bx, (int)d->nbx[f.ci], sm, decision); break;
#define AB_FUSED_COL_K(LH) AB_FUSED_COL(LH, 2, 1) AB_FUSED_COL(LH, 3, 2) AB_FUSED_COL(LH, 4, 2) AB_FUSED_COL(LH, 5, 4)

__global__ void __launch_bounds__(COL_THREADS, 2) k_fused_colpass(const FusedColPass * __restrict__ d, const TConst * __restrict__ tcs)
{
	extern __shared__ __align__(16) u32 sm[];
	__shared__ TConst cs;
	__shared__ int decision;
	const FusedCta f = fused_cta(d, blockIdx.x);
	const ColJob J = d->jobs[f.ci].j[f.job];
	const u32 amul = (J.mult != nullptr) ? J.mult[f.cand] : J.a;
	if (amul == 0u) return;                       // inactive batch slot
	fused_consts(cs, tcs, f.ci);
	switch (d->sel[f.ci])
	{
	AB_FUSED_COL_K(1) AB_FUSED_COL_K(2) AB_FUSED_COL_K(3) AB_FUSED_COL_K(4) AB_FUSED_COL_K(5) AB_FUSED_COL_K(6)
	default: break;
	}
}
#undef AB_FUSED_COL_K
#undef AB_FUSED_COL

// ================================================================ register words of the reference
// Canonical residue of the exact value (d0, d1, d2) mod a reference prime:
// d0 + d1 2^32 + d2 2^64 with Montgomery steps (r2 = 2^64 mod p, so
// ref_mont(x, r2) = x 2^32 mod p); a negative value is negated first.
__device__ __forceinline__ u32 ref_mont(u32 a, u32 b, u32 p, u32 q)
{
	const u64 t = (u64)a * b;
	const u32 m = (u32)t * q;
	return ref_sub((u32)(t >> 32), __umulhi(m, p), p);
}

__device__ __forceinline__ u32 ref_add(u32 a, u32 b, u32 p) { return ref_sub(a, p - b, p); }

// Both conversions take one register, or two with interleaved planes of words
// (plane k of the second after plane k of the first: a checkpoint's payload),
// blockIdx.y the register, ws the words between planes.
__global__ void k_export(const RefConst rc, const u32 * __restrict__ norm0, const u32 * __restrict__ norm1, u32 * __restrict__ words, u32 n, u32 ws)
{
	const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
	griddep_wait();
	if (i >= n) return;
	const u32 * __restrict__ norm = (blockIdx.y == 0) ? norm0 : norm1;
	words += blockIdx.y * n;
	u32 d0 = norm[i], d1 = norm[n + i], d2 = norm[2 * (size_t)n + i];
	const bool neg = (i32)d2 < 0;
	if (neg)
	{
		// two's-complement negation of the 96-bit value
		d0 = ~d0; d1 = ~d1; d2 = ~d2;
		d0 += 1; if (d0 == 0) { d1 += 1; if (d1 == 0) d2 += 1; }
	}
	for (int k = 0; k < rc.K; ++k)
	{
		const u32 p = rc.p[k], q = rc.q[k], r2 = rc.r2[k];
		const u32 a0 = ref_red(d0, p);
		const u32 a1 = ref_mont(d1, r2, p, q);                       // d1 2^32
		const u32 a2 = ref_mont(ref_mont(d2, r2, p, q), r2, p, q);   // d2 2^64
		u32 r = ref_add(ref_add(a0, a1, p), a2, p);
		if (neg && r != 0) r = p - r;
		words[(size_t)k * ws + i] = r;
	}
}

// Exact signed value from the K residues (mixed-radix Garner, leading digit
// balanced; kernel.cl:1231-1470), checked against the 96-bit normal form.
template <int K>
__global__ void k_import(const RefConst rc, const u32 * __restrict__ words, u32 * __restrict__ norm0, u32 * __restrict__ norm1, u32 n, u32 ws, u32 * bad)
{
	const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
	griddep_wait();
	if (i >= n) return;
	u32 * __restrict__ norm = (blockIdx.y == 0) ? norm0 : norm1;
	words += blockIdx.y * n;
	u32 u[K];
#pragma unroll
	for (int ii = K - 1; ii >= 0; --ii)
	{
		u32 v = words[(size_t)ii * ws + i];
#pragma unroll
		for (int j = K - 1; j > ii; --j) v = ref_mont_c(ref_sub(v, u[j], rc.p[ii]), rc.gm[ii][j], rc.gmq[ii][j], rc.p[ii]);
		u[ii] = v;
	}
	const i32 i0 = (u[0] > (rc.p[0] >> 1)) ? (i32)(u[0] - rc.p[0]) : (i32)u[0];
	Big<K> V;
	{
		const i64 v01 = (i64)i0 * (i64)rc.p[1] + (i64)u[1];
		V.l[0] = (u32)v01; V.l[1] = (u32)((u64)v01 >> 32);
		const u32 sgn = (v01 < 0) ? 0xffffffffu : 0u;
#pragma unroll
		for (int l = 2; l < K; ++l) V.l[l] = sgn;
	}
#pragma unroll
	for (int l = 2; l < K; ++l) V = big_add_u32<K>(big_mul_u32<K>(V, rc.p[l]), u[l]);
	const u32 sgn = big_is_neg<K>(V) ? 0xffffffffu : 0u;
	u32 x[AB_NW];
#pragma unroll
	for (int l = 0; l < AB_NW; ++l) x[l] = (l < K) ? V.l[l] : sgn;
	bool fits = (K < AB_NW) || (((i32)x[2] < 0) == (sgn != 0));
#pragma unroll
	for (int l = AB_NW; l < K; ++l) fits = fits && (V.l[l] == sgn);
	if (!fits) atomicOr(bad, 1u);
#pragma unroll
	for (int l = 0; l < AB_NW; ++l) norm[(size_t)l * n + i] = x[l];
}

// ================================================================ mid pass
// The G levels between the column and the row levels (lengths above 2^20):
// with i = (h 2^G + m) R + c, global level LA + t works on bit G-1-t of m,
// block j = h 2^t + (m >> (G - t)).  One thread per (prime, h, c): 2^G words
// at stride R (consecutive threads, consecutive c).  Forward: [0, 4p) in and
// out; inverse: [0, 2p), twiddles -w^-1 (domain Q: the mirrored w).
template <int G, bool INV>
__global__ void __launch_bounds__(256) k_midpass(const RowJobs jobs, const TConst c)
{
	constexpr int M = 1 << G;
	const RowJob J = (blockIdx.y == 0) ? jobs.j[0] : jobs.j[1];
	const u32 cand = blockIdx.z;
	if (J.active != nullptr && J.active[cand] == 0u) return;
	const u32 R = c.R >> G;                      // row-pass row length
	const u32 per = c.H * R;
	const u32 gid = blockIdx.x * blockDim.x + threadIdx.x;
	if (gid >= (u32)c.KP * per) return;
	const u32 k = gid / per, rem = gid - k * per, h = rem / R, col = rem - h * R;
	const u32 p = c.p[k], p2 = 2 * p;
	u32 * __restrict__ x = J.x + (size_t)cand * J.stride + (size_t)k * c.n + (size_t)h * M * R + col;
	const uint2 * __restrict__ w = J.w + (size_t)k * (c.n >> 1);
	const uint2 * __restrict__ wi = (J.wi != nullptr) ? J.wi + (size_t)k * (c.n >> 1) : nullptr;
	griddep_wait();
	u32 v[M];
#pragma unroll
	for (int m = 0; m < M; ++m) v[m] = x[(size_t)m * R];
#pragma unroll
	for (int tt = 0; tt < G; ++tt)
	{
		const int t = INV ? G - 1 - tt : tt;
		const int half = M >> (t + 1);
		const u32 lvl = 1u << (c.LA + t);
#pragma unroll
		for (int blk = 0; blk < (1 << t); ++blk)
		{
			const u32 idx = lvl + (h << t) + (u32)blk;
			const uint2 wv = !INV ? __ldg(w + idx) : (wi != nullptr) ? __ldg(wi + idx) : __ldg(w + (3u * lvl - 1u - idx));
#pragma unroll
			for (int q = 0; q < half; ++q)
			{
				const int m0 = blk * 2 * half + q;
				if (INV) inv_bf(v[m0], v[m0 + half], wv.x, wv.y, p, p2);
				else fwd_bf(v[m0], v[m0 + half], wv.x, wv.y, p, p2);
			}
		}
	}
#pragma unroll
	for (int m = 0; m < M; ++m) x[(size_t)m * R] = v[m];
}

// ================================================================ host side
bool make_geometry(int ln, int lb_override, Geometry & g)
{
	if (ln < 6 || ln > 22) return false;
	const int L = ln - 1;
	// default split, measured on B200 over every split (ln 13..20, single
	// transforms; batches agree): us per squaring, e.g. ln 13 LB 9 / 10: 20.7 /
	// 21.0 and, 32 slots, 51.8 / 62.2 per step; ln 15 LB 10 / 11: 28.2 / 26.9; ln 17
	// LB 10 / 11: 48.4 / 48.1; ln 18 LB 11 / 12: 82.6 / 90.8.  Above 2^20 the row
	// and column passes are full (13 and 6 levels) and the mid pass takes the 1
	// or 2 levels left.
	static const int DEFAULT_LB[23] = {0, 0, 0, 0, 0, 0, 4, 4, 5, 6, 7, 8, 9, 9, 10, 11, 11, 11, 11, 12, 13, 13, 13};
	int LB = (lb_override > 0) ? lb_override : DEFAULT_LB[ln];
	if (lb_override <= 0 && L - LB > 6 && ln <= 20) LB = L - 6;
	if (LB < 4 || LB > 13 || LB > L - 1) return false;
	const int LA = (L - LB < 6) ? L - LB : 6, G = L - LB - LA;
	if (G > 3) return false;
	g.ln = ln; g.LB = LB; g.LA = LA; g.G = G;
	g.H = 1u << LA; g.R = 1u << (LB + 1); g.HR = g.H << G; g.RC = g.R << G; g.NC = col_ctas(g.RC);
	return true;
}

size_t colpass_smem(const Geometry & g, int KP)
{
	const size_t L = (size_t)KP - 1;
	return sizeof(u32) * ((size_t)KP * g.H * CW + (size_t)g.H * 8 * L + 24) + sizeof(uint2) * 3 * (size_t)KP * g.H;
}

template <int LOG_R, int MODE>
static cudaError_t rowpass_m(const Geometry & g, const TConst & c, const RowJobs & jobs, int njobs, cudaStream_t s, int ncand)
{
	const size_t smem = RowCfg<LOG_R>::SMEM;
	static std::atomic<unsigned long long> attr_done{0};
	const cudaError_t e = allow_dynamic_smem(k_rowpass<LOG_R, MODE>, smem, attr_done);
	if (e != cudaSuccess) return e;
	if (ncand == 0) return cudaSuccess;      // set-up only (before a stream capture)
	const dim3 grid((unsigned)(c.KP * g.HR), (unsigned)njobs, (unsigned)ncand);
	return launch_pdl(k_rowpass<LOG_R, MODE>, grid, dim3(RowCfg<LOG_R>::NT), smem, s, jobs, c);
}

// The jobs of a launch have one mode.
template <int LOG_R>
static cudaError_t rowpass_t(const Geometry & g, const TConst & c, const RowJobs & jobs, int njobs, cudaStream_t s, int ncand)
{
	if (ncand == 0)
	{
		cudaError_t e = rowpass_m<LOG_R, ROW_FWD_ONLY>(g, c, jobs, njobs, s, 0);
		if (e == cudaSuccess) e = rowpass_m<LOG_R, ROW_SQUARE>(g, c, jobs, njobs, s, 0);
		return (e != cudaSuccess) ? e : rowpass_m<LOG_R, ROW_MUL>(g, c, jobs, njobs, s, 0);
	}
	if (njobs > 1 && jobs.j[1].mode != jobs.j[0].mode) return cudaErrorInvalidValue;
	switch (jobs.j[0].mode)
	{
	case ROW_FWD_ONLY: return rowpass_m<LOG_R, ROW_FWD_ONLY>(g, c, jobs, njobs, s, ncand);
	case ROW_SQUARE: return rowpass_m<LOG_R, ROW_SQUARE>(g, c, jobs, njobs, s, ncand);
	case ROW_MUL: return rowpass_m<LOG_R, ROW_MUL>(g, c, jobs, njobs, s, ncand);
	default: return cudaErrorInvalidValue;
	}
}

cudaError_t launch_rowpass(const Geometry & g, const TConst & c, const RowJobs & jobs, int njobs, cudaStream_t s, int ncand)
{
	switch (g.LB + 1)
	{
	case 5: return rowpass_t<5>(g, c, jobs, njobs, s, ncand);
	case 6: return rowpass_t<6>(g, c, jobs, njobs, s, ncand);
	case 7: return rowpass_t<7>(g, c, jobs, njobs, s, ncand);
	case 8: return rowpass_t<8>(g, c, jobs, njobs, s, ncand);
	case 9: return rowpass_t<9>(g, c, jobs, njobs, s, ncand);
	case 10: return rowpass_t<10>(g, c, jobs, njobs, s, ncand);
	case 11: return rowpass_t<11>(g, c, jobs, njobs, s, ncand);
	case 12: return rowpass_t<12>(g, c, jobs, njobs, s, ncand);
	case 13: return rowpass_t<13>(g, c, jobs, njobs, s, ncand);
	case 14: return rowpass_t<14>(g, c, jobs, njobs, s, ncand);
	default: return cudaErrorInvalidValue;
	}
}

template <int G>
static cudaError_t midpass_t(const Geometry & g, const TConst & c, const RowJobs & jobs, int njobs, cudaStream_t s, int ncand, bool inverse)
{
	const u32 threads = (u32)c.KP * g.H * g.R;
	const dim3 grid((threads + 255) / 256, (unsigned)njobs, (unsigned)ncand);
	if (inverse) return launch_pdl(k_midpass<G, true>, grid, dim3(256), 0, s, jobs, c);
	return launch_pdl(k_midpass<G, false>, grid, dim3(256), 0, s, jobs, c);
}

cudaError_t launch_midpass(const Geometry & g, const TConst & c, const RowJobs & jobs, int njobs, cudaStream_t s, int ncand, bool inverse)
{
	if (ncand == 0) return cudaSuccess;
	switch (g.G)
	{
	case 1: return midpass_t<1>(g, c, jobs, njobs, s, ncand, inverse);
	case 2: return midpass_t<2>(g, c, jobs, njobs, s, ncand, inverse);
	case 3: return midpass_t<3>(g, c, jobs, njobs, s, ncand, inverse);
	default: return cudaErrorInvalidValue;
	}
}

cudaError_t launch_colpass2(const Geometry & g, const TConst & c, const ColJobs & jobs, int njobs, cudaStream_t s, int ncand);
cudaError_t launch_colpass3(const Geometry & g, const TConst & c, const ColJobs & jobs, int njobs, cudaStream_t s, int ncand);
cudaError_t launch_colpass4(const Geometry & g, const TConst & c, const ColJobs & jobs, int njobs, cudaStream_t s, int ncand);
cudaError_t launch_colpass5(const Geometry & g, const TConst & c, const ColJobs & jobs, int njobs, cudaStream_t s, int ncand);

cudaError_t launch_colpass(const Geometry & g, const TConst & c, const ColJobs & jobs, int njobs, cudaStream_t s, int ncand)
{
	switch (c.K)
	{
	case 2: return launch_colpass2(g, c, jobs, njobs, s, ncand);
	case 3: return launch_colpass3(g, c, jobs, njobs, s, ncand);
	case 4: return launch_colpass4(g, c, jobs, njobs, s, ncand);
	case 5: return launch_colpass5(g, c, jobs, njobs, s, ncand);
	default: return cudaErrorInvalidValue;
	}
}

size_t fused_rowpass_smem(int log_r)
{
	return sizeof(u32) * (((size_t)1 << log_r) + ((size_t)1 << log_r) / 16);
}

cudaError_t launch_fused_rowpass(const FusedRowPass * d, const TConst * tcs, u32 ctas, size_t smem, cudaStream_t s)
{
	static std::atomic<unsigned long long> attr_done{0};
	static size_t set_smem = 0;
	if (smem > set_smem)
	{
		attr_done.store(0);
		set_smem = smem;
	}
	const cudaError_t e = allow_dynamic_smem(k_fused_rowpass, set_smem, attr_done);
	if (e != cudaSuccess || ctas == 0) return e;
	return launch_pdl(k_fused_rowpass, dim3(ctas), dim3(AB_FUSED_ROW_THREADS), smem, s, d, tcs);
}

cudaError_t launch_fused_colpass(const FusedColPass * d, const TConst * tcs, u32 ctas, size_t smem, cudaStream_t s)
{
	static std::atomic<unsigned long long> attr_done{0};
	static size_t set_smem = 0;
	if (smem > set_smem)
	{
		attr_done.store(0);
		set_smem = smem;
	}
	const cudaError_t e = allow_dynamic_smem(k_fused_colpass, set_smem, attr_done);
	if (e != cudaSuccess || ctas == 0) return e;
	return launch_pdl(k_fused_colpass, dim3(ctas), dim3(COL_THREADS), smem, s, d, tcs);
}

cudaError_t launch_export(const RefConst & rc, const u32 * norm0, const u32 * norm1, u32 * words, u32 n, cudaStream_t s)
{
	if (n == 0) return cudaSuccess;
	const u32 regs = (norm1 != nullptr) ? 2 : 1;
	return launch_pdl(k_export, dim3((n + 255) / 256, regs), dim3(256), 0, s, rc, norm0, norm1, words, n, regs * n);
}

template <int K>
static cudaError_t import_t(const RefConst & rc, const u32 * words, u32 * norm0, u32 * norm1, u32 n, u32 * bad, cudaStream_t s)
{
	const u32 regs = (norm1 != nullptr) ? 2 : 1;
	return launch_pdl(k_import<K>, dim3((n + 255) / 256, regs), dim3(256), 0, s, rc, words, norm0, norm1, n, regs * n, bad);
}

cudaError_t launch_import(const RefConst & rc, const u32 * words, u32 * norm0, u32 * norm1, u32 n, u32 * bad, cudaStream_t s)
{
	if (n == 0) return cudaSuccess;
	switch (rc.K)
	{
	case 2: return import_t<2>(rc, words, norm0, norm1, n, bad, s);
	case 3: return import_t<3>(rc, words, norm0, norm1, n, bad, s);
	case 4: return import_t<4>(rc, words, norm0, norm1, n, bad, s);
	case 5: return import_t<5>(rc, words, norm0, norm1, n, bad, s);
	default: return cudaErrorInvalidValue;
	}
}

} // namespace ab
