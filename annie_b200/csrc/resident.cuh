// Short transforms (up to 2^12 words per prime), resident in shared memory.
//
// One thread-block cluster holds one candidate for a whole run of squarings:
// CTA dom KP + k keeps the transform of prime k in domain dom (0 = R, 1 = Q)
// in its shared memory, with the twiddles and the image of N^-1 (R) or N (Q).
// A squaring is three products; each is a transform step inside every CTA
// (forward levels, pointwise product, inverse levels) and a carry step over
// coefficients, in which every CTA gathers the residues of its range from the
// others (distributed shared memory), carries, and writes the new residues
// into the CTAs of the next product.  A hardware cluster barrier separates the
// steps: six per squaring, where the row and column passes need six dependent
// kernel launches and the L2 between them.  Those short launches cost 3 to
// 5 us each whatever the length; the cluster's steps cost what their longest
// dependency chain costs.  B200, us per squaring, passes then / resident: 2,500
// bits 22.6 / 5.9, 20k 25.3 / 7.3, 60k 33.3 / 10.0, 100k 28.5 / 12.1, 262k 34.7 /
// 18.5 (the passes as they are now: 262k 21.9).  At 2^12 words a transform step
// takes 7 k to 8 k clocks (multiplier floor 3.5 k) and a carry step 4.5 k.
//
// The arithmetic is that of the passes (kernels.cu): the same primes, twiddle
// positions, products, CRT and carry rule, so the registers are the same.
#pragma once
#include <atomic>
#include <type_traits>

#include "kernels.h"
#include "carry.cuh"
#include "levels.cuh"
#include "pdl.cuh"

namespace ab
{

namespace
{

__device__ __forceinline__ u32 cluster_rank()
{
	u32 r;
	asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
	return r;
}

// All threads of the cluster; orders shared-memory accesses of all its CTAs.
__device__ __forceinline__ void cluster_sync()
{
	__syncwarp();
	asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Address of this CTA's shared variable at p, in CTA `rank` of the cluster.
__device__ __forceinline__ u32 remote(const void * p, u32 rank)
{
	u32 r;
	asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((u32)__cvta_generic_to_shared(p)), "r"(rank));
	return r;
}
__device__ __forceinline__ u32 ld_remote(u32 a)
{
	u32 v;
	asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
	return v;
}
__device__ __forceinline__ void st_remote(u32 a, u32 v)
{
	asm volatile("st.shared::cluster.u32 [%0], %1;" :: "r"(a), "r"(v) : "memory");
}

constexpr u32 RES_THREADS = 1024;                       // of an SM that a kernel is compiled for (64 registers each)
template <int LN, int K>
struct ResCfg
{
	static constexpr int KP = K + 1, C = 2 * KP;               // CTAs of a cluster
	static constexpr u32 N = 1u << LN, G = N / 4;              // words, groups of 4 coefficients
	// groups of a CTA in the carry steps: of a Q CTA where those carry T_Q alone
	static constexpr u32 Q = (G + C - 1) / C, Q2 = (G + KP - 1) / KP;
	// threads: 8 words each in a transform step; in a carry step a lane per
	// coefficient, with up to two predecessor groups
	static constexpr u32 NC = ((Q + 2) * 4 + 31) / 32 * 32;
	static constexpr u32 NT0 = (N / 8 > NC) ? N / 8 : NC, NT = (NT0 < 64) ? 64 : (NT0 + 31) / 32 * 32;
	static constexpr u32 CH = NT / 4 - 1;                      // groups of T_Q carried at a time
	// shared memory, words: two work buffers; the operand's image; the second
	// factor's, or m' of a sparse N; the twiddles; the inverse twiddles (R), or
	// T_Q (Q); carries
	static constexpr u32 W = rpad(N);
	static constexpr u32 TQ = Q2 * 4 * AB_NW, MQ = Q * 4 * AB_NW, CWN = NT / 4 * K;
	static constexpr size_t SMEM = sizeof(u32) * (2 * W + 3 * N + (N > TQ ? N : TQ) + CWN);
	static_assert(MQ <= N, "m' in the second factor's place");
	// CTAs per SM that the kernel is compiled for
	static constexpr u32 BY_T = RES_THREADS / NT, BY_S = (u32)((size_t)227 * 1024 / (SMEM + 1024));
	static constexpr u32 MINB = (BY_T < BY_S ? BY_T : BY_S) < 1 ? 1 : (BY_T < BY_S ? BY_T : BY_S);
};

// One transform step of a CTA: the residues in xb, forward, product with the
// image op, inverse into xa; or (BOTTOM_FORWARD) the image into op.  op: two
// planes of N/8 uint4 (a thread's 8 words, without bank conflicts).
template <int LN>
__device__ __forceinline__ void res_transform(const u32 * xb, u32 * xa, u32 * op, int mode, const LevelTw & tw, u32 p, u32 pinv)
{
	uint4 * const q = reinterpret_cast<uint4 *>(op);
	constexpr u32 N8 = (1u << LN) / 8;
	level_transform<LN>(xb, xa, mode, tw, threadIdx.x, blockDim.x, p, pinv,
		[&](u32 o, uint4 & a, uint4 & b) { a = q[o]; b = q[N8 + o]; },
		[&](u32 o, uint4 a, uint4 b) { q[o] = a; q[N8 + o] = b; });
}

// Groups g0 .. g0 + cnt - 1 of a carry step, and the E predecessor groups that
// give the carry into them (the groups before 0 end the register).
struct CarryRange
{
	u32 g0, cnt, E;
};

// An exact value that the CTAs from `first` on keep, QQ groups each, as three
// planes of 4 QQ words.
template <u32 QQ>
__device__ __forceinline__ void get_exact(const u32 * planes, u32 first, u32 i, u32 & d0, u32 & d1, u32 & d2)
{
	const u32 own = (i >> 2) / QQ, a = remote(planes, first + own) + (u32)sizeof(u32) * (i - own * 4 * QQ);
	d0 = ld_remote(a);
	d1 = ld_remote(a + (u32)sizeof(u32) * 4 * QQ);
	d2 = ld_remote(a + 2 * (u32)sizeof(u32) * 4 * QQ);
}

// The carry of one product over a range, a lane per coefficient and 4 lanes per
// group, the predecessor groups first (CTA 0 has two when it re-derives the
// register's last coefficient for the mod R / mod Q decision).  The product's
// residues are in xa of the CTAs from src on; with mq, it is that of the sparse
// N with the exact values there.  tq: subtract T_Q.  Returns the coefficient's
// exact value in x and whether the lane owns it.
template <int LN, int K, int PCK, bool FULL>
__device__ __forceinline__ bool res_carry(const TConst & c, const CarryRange & rg, u32 src, bool nega, u32 amul, const u32 * tq, int lower,
	const Width & w, int wbits, const u32 * xa, const SparseN * sp, const u32 * mq, u32 * cw, int * decision, u32 (&x)[AB_NW], u32 & e)
{
	using Cfg = ResCfg<LN, K>;
	constexpr int KP = Cfg::KP, L = K, ND = DigitLimbs<PCK>::N;
	constexpr u32 G = Cfg::G, N = Cfg::N;
	const u32 E = rg.E, li = threadIdx.x >> 2, j = threadIdx.x & 3;
	const bool active = li < E + rg.cnt;
	const u32 g = rg.g0 + li - E + ((rg.g0 + li < E) ? G : 0u);
	e = active ? 4 * g + j : 0u;
	Big<L> f = big_zero<L>();
	if (active)
	{
		u32 y[KP] = {};
		if (mq == nullptr)
		{
			const u32 o = (u32)sizeof(u32) * rpad(e);
#pragma unroll
			for (int k = 0; k < KP; ++k) y[k] = ld_remote(remote(xa, src + k) + o);
		}
		u32 s[AB_NW];
		if (tq != nullptr) get_exact<Cfg::Q2>(tq, KP, e, s[0], s[1], s[2]);
		if (mq != nullptr) f = sparse_product<L>(*sp, e, N, [&](u32 i, u32 & d0, u32 & d1, u32 & d2) { get_exact<Cfg::Q>(mq, 0, i, d0, d1, d2); });
		else f = crt<L>(c, y);
		if (amul != 1u) f = big_mul_u32<L>(f, amul);
		if (tq != nullptr) f = big_sub<L>(f, big_from_exact<L>(s[0], s[1], s[2]));
	}
	// phase 1: the group's digits and carry-out
	u32 d[ND];
	lane_digits<FULL, L, ND>(f, w, j, d);
	if (active && j == 3)
	{
#pragma unroll
		for (int l = 0; l < L; ++l) cw[li * L + l] = f.l[l];
	}
	__syncthreads();
	// phase 2: the previous group's carry-out, balanced digits; the last
	// coefficient of a group absorbs the rest
	const bool top0 = (lower != LOWER_NONE) && E == 2 && li == 1;
	const bool mine = active && li >= E;
	Big<L> cin = big_zero<L>();
	if (j == 0 && (mine || top0))
	{
#pragma unroll
		for (int l = 0; l < L; ++l) cin.l[l] = cw[(li - 1) * L + l];
		if (g == 0 && nega) cin = big_neg<L>(cin);
	}
	lane_balance<FULL, L, ND>(cin, d, w, half_of(wbits), j, x);
	if (lower != LOWER_NONE)
	{
		// mod R (+2) / mod Q on the top and bottom coefficients (kernel.cl:1653-1683):
		// whether the last coefficient is 2^W or more.  The step is written out here
		// and twice in the column pass: one function for all three measured slower
		// (us per squaring: 20k bits 7.26 -> 7.50, 6.6M bits 47.9 -> 48.7).
		if ((mine || top0) && e == N - 1) *decision = reaches_width(x, w) ? 1 : 0;
		__syncthreads();
		if (mine && (e == 0 || e == N - 1))
		{
			Big<AB_NW> a, b;
#pragma unroll
			for (int i = 0; i < AB_NW; ++i) a.l[i] = x[i];
			if (e == 0)
			{
				int dv = 0;
				if (*decision) dv += (lower == LOWER_Q) ? -1 : 1;
				if (lower == LOWER_R_ADD2) dv += 2;
				b.l[0] = (u32)dv; b.l[1] = b.l[2] = (u32)(dv >> 31);
				a = big_add<AB_NW>(a, b);
			}
			else if (*decision)
			{
#pragma unroll
				for (int i = 0; i < AB_NW; ++i) b.l[i] = (i == (wbits >> 5)) ? 1u << (wbits & 31) : 0u;
				a = big_sub<AB_NW>(a, b);
			}
#pragma unroll
			for (int i = 0; i < AB_NW; ++i) x[i] = a.l[i];
		}
	}
	return mine;
}

// SOLO: a launch of one cluster, which needs no other resident beside it and
// may use all registers (262k bits: 18.5 us per squaring against 19.5).
template <int LN, int K, int PCK, bool SOLO>
__global__ void __launch_bounds__(ResCfg<LN, K>::NT, SOLO ? 1 : ResCfg<LN, K>::MINB) k_resident(const ResJob J, const TConst c)
{
	using Cfg = ResCfg<LN, K>;
	constexpr int KP = Cfg::KP;
	constexpr u32 N = Cfg::N, W = Cfg::W, G = Cfg::G;
	extern __shared__ __align__(16) u32 sm[];
	__shared__ int decision;
	u32 * const xa = sm, * const xb = xa + W;               // transform step: xb -> xa
	u32 * const op = xb + W;                                // image of N^-1 (R) or N (Q)
	u32 * const op2 = op + N;                               // image of the second factor of a product
	u32 * const mq = op2;                                   // m' of a CTA's range when N is sparse, planes of 4 Q words
	uint2 * const w = reinterpret_cast<uint2 *>(op2 + N);
	uint2 * const wi = w + N / 2;                           // R CTAs
	u32 * const tq = reinterpret_cast<u32 *>(wi);           // Q CTAs: T_Q of the CTA's range, planes of 4 Q2 words
	u32 * const cw = reinterpret_cast<u32 *>(wi) + (N > Cfg::TQ ? N : Cfg::TQ);

	const u32 rank = cluster_rank(), cand = blockIdx.y;
	const u32 dom = rank / KP, k = rank - dom * KP;
	const u32 tid = threadIdx.x, NT = Cfg::NT;
	const u32 p = c.p[k], pinv = c.pinv[k];
	const size_t on = (size_t)cand * J.stride_norm, ot = (size_t)cand * J.stride_ntt;
	u32 * const reg = J.reg + on;
	const uint2 * const gw = (dom == 0 ? J.wr : J.wq) + (size_t)k * (N / 2);
	for (u32 i = tid; i < N / 2; i += NT)
	{
		w[i] = __ldg(gw + i);
		if (dom == 0) wi[i] = __ldg(J.wri + (size_t)k * (N / 2) + i);
	}
	const LevelTw tw{ w, wi, dom != 0 };
	{
		const uint4 * img = reinterpret_cast<const uint4 *>((dom == 0 ? J.nir : J.nq) + ot + (size_t)k * N);
		uint4 * o4 = reinterpret_cast<uint4 *>(op);
		for (u32 i = tid; i < N / 4; i += NT) o4[(i & 1) * (N / 8) + (i >> 1)] = __ldg(img + i);
	}
	__shared__ SparseN sp;
	if (tid == 0) sp = J.cand[cand].sp;
	const int wbits = PCK * J.cand[cand].lbase;
	// above: tables and images, which no earlier work of the stream writes
	griddep_wait();
	// the last step that the slot takes part in; an idle slot's cluster leaves
	__shared__ int last;
	if (tid == 0) last = (J.mult != nullptr) ? -1 : J.steps - 1;
	__syncthreads();
	if (J.mult != nullptr)
	{
		for (int s = (int)tid; s < J.steps; s += (int)NT)
			if (J.mult[(size_t)s * J.ctrl_stride + cand] != 0u) atomicMax(&last, s);
		__syncthreads();
		if (last < 0) return;
	}
	auto encode_all = [&](const u32 * src) {
		const uint4 * s0 = reinterpret_cast<const uint4 *>(src), * s1 = s0 + N / 4, * s2 = s1 + N / 4;
		for (u32 i = tid; i < N / 4; i += NT)
		{
			const uint4 a = s0[i], b = s1[i], d = s2[i];
			*reinterpret_cast<uint4 *>(xb + rpad(4 * i)) = make_uint4(
				encode_res(c, (int)k, a.x, b.x, d.x), encode_res(c, (int)k, a.y, b.y, d.y),
				encode_res(c, (int)k, a.z, b.z, d.z), encode_res(c, (int)k, a.w, b.w, d.w));
		}
	};
	if (J.y != nullptr)
	{
		encode_all(J.y + on);
		__syncthreads();
		res_transform<LN>(xb, xa, op2, BOTTOM_FORWARD, tw, p, pinv);
		__syncthreads();
	}
	encode_all(reg);
	__syncthreads();

	const bool sparse = (sp.nt != 0u);
	const Width wd = make_width(wbits);
	const bool full = (wd.ws == DigitLimbs<PCK>::N - 1);
	auto carry = [&](const CarryRange & rg, u32 src, bool nega, u32 amul, const u32 * sub, int lower, const u32 * m, u32 (&x)[AB_NW], u32 & e) {
		return full ? res_carry<LN, K, PCK, true>(c, rg, src, nega, amul, sub, lower, wd, wbits, xa, &sp, m, cw, &decision, x, e)
		            : res_carry<LN, K, PCK, false>(c, rg, src, nega, amul, sub, lower, wd, wbits, xa, &sp, m, cw, &decision, x, e);
	};
	// the CTA's groups: of all carry steps but that of T_Q, and of T_Q (Q CTAs)
	const u32 g0 = rank * Cfg::Q, cnt = (g0 >= G) ? 0u : (G - g0 < Cfg::Q) ? G - g0 : Cfg::Q;
	const CarryRange own{ g0, cnt, (cnt == 0) ? 0u : (rank == 0) ? 2u : 1u };
	const u32 q0 = (rank - dom * KP) * Cfg::Q2, qn = (q0 >= G) ? 0u : (G - q0 < Cfg::Q2) ? G - q0 : Cfg::Q2;
	// residues of a coefficient into the CTAs of domain d
	auto scatter = [&](const u32 (&x)[AB_NW], u32 e, bool r_dom, bool q_dom) {
		const u32 o = (u32)sizeof(u32) * rpad(e);
#pragma unroll
		for (int q = 0; q < KP; ++q)
		{
			const u32 v = encode_res(c, q, x[0], x[1], x[2]);
			if (r_dom) st_remote(remote(xb, (u32)q) + o, v);
			if (q_dom) st_remote(remote(xb, (u32)(KP + q)) + o, v);
		}
	};
#pragma unroll 1
	for (int s = 0; s < J.steps; ++s)
	{
		const u32 amul = (J.mult != nullptr) ? J.mult[(size_t)s * J.ctrl_stride + cand] : ((J.bits >> s) & 1) ? J.a : 1u;
		if (amul == 0u) continue;                 // the slot rests in this step
		if (s == last && gridDim.y == 1) griddep_launch();   // the next run may load its tables
		u32 x[AB_NW], e;
		// T_R = a x y mod R, T_Q = a x y mod Q
		res_transform<LN>(xb, xa, op2, (J.y != nullptr) ? BOTTOM_MUL : BOTTOM_SQUARE, tw, p, pinv);
		cluster_sync();
		if (carry(own, 0u, false, amul, nullptr, LOWER_NONE, nullptr, x, e)) scatter(x, e, true, false);
		cluster_sync();
		// m' = T_R N^-1 mod R, + 2; meanwhile the Q CTAs carry T_Q, which is only
		// needed at the end
		if (dom == 0) res_transform<LN>(xb, xa, op, BOTTOM_MUL, tw, p, pinv);
		else
		{
#pragma unroll 1
			for (u32 i = 0; i < qn; i += Cfg::CH)
			{
				if (i != 0) __syncthreads();
				const CarryRange rg{ q0 + i, (qn - i < Cfg::CH) ? qn - i : Cfg::CH, 1u };
				if (carry(rg, (u32)KP, true, amul, nullptr, LOWER_NONE, nullptr, x, e))
				{
#pragma unroll
					for (int l = 0; l < AB_NW; ++l) tq[l * 4 * Cfg::Q2 + e - 4 * q0] = x[l];
				}
			}
		}
		cluster_sync();
		if (carry(own, 0u, false, 1u, nullptr, LOWER_R_ADD2, nullptr, x, e))
		{
			if (sparse)
			{
#pragma unroll
				for (int l = 0; l < AB_NW; ++l) mq[l * 4 * Cfg::Q + e - 4 * g0] = x[l];
			}
			else scatter(x, e, false, true);
		}
		cluster_sync();
		// m' N - T_Q mod Q: a sparse N needs no transform
		if (!sparse)
		{
			if (dom == 1) res_transform<LN>(xb, xa, op, BOTTOM_MUL, tw, p, pinv);
			cluster_sync();
		}
		const bool snap = (J.snap != nullptr) && J.snap[(size_t)s * J.ctrl_stride + cand] != 0u;
		if (carry(own, (u32)KP, true, 1u, tq, LOWER_Q, sparse ? mq : nullptr, x, e))
		{
			scatter(x, e, true, true);
#pragma unroll
			for (u32 l = 0; l < AB_NW; ++l)
			{
				if (s == last) reg[l * N + e] = x[l];
				if (snap) J.out_snap[on + l * N + e] = x[l];
			}
		}
		cluster_sync();
	}
}

template <int LN, int K, int PCK, bool SOLO>
cudaError_t resident_v(const ResJob & J, const TConst & c, cudaStream_t s, int ncand, bool * fits)
{
	using Cfg = ResCfg<LN, K>;
	static_assert(Cfg::NC <= 1024 && Cfg::NT <= 1024, "a lane per coefficient");
	// per device: the kernel's attributes, and whether a cluster of it fits
	static std::atomic<unsigned long long> done{0}, ok{0};
	int dev = 0;
	cudaError_t e = cudaGetDevice(&dev);
	if (e != cudaSuccess) return e;
	const unsigned long long bit = 1ull << (dev & 63);
	cudaLaunchConfig_t cfg = {};
	cfg.gridDim = dim3(Cfg::C, (unsigned)ncand);
	cfg.blockDim = dim3(Cfg::NT);
	cfg.dynamicSmemBytes = Cfg::SMEM;
	cfg.stream = s;
	cudaLaunchAttribute attr[2];
	attr[0].id = cudaLaunchAttributeClusterDimension;
	attr[0].val.clusterDim.x = Cfg::C;
	attr[0].val.clusterDim.y = 1;
	attr[0].val.clusterDim.z = 1;
	attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
	attr[1].val.programmaticStreamSerializationAllowed = 1;
	cfg.attrs = attr;
	// a run of several clusters starts after the one before: placed among its
	// last ones, fewer clusters fit (16 x 262k bits: 57 us per step against 32)
	cfg.numAttrs = (ncand == 1) ? 2 : 1;
	if (!(done.load(std::memory_order_acquire) & bit))
	{
		e = cudaFuncSetAttribute(k_resident<LN, K, PCK, SOLO>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg::SMEM);
		if (e != cudaSuccess) return e;
		if (Cfg::C > 8) e = cudaFuncSetAttribute(k_resident<LN, K, PCK, SOLO>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
		if (e != cudaSuccess) return e;
		cfg.gridDim = dim3(Cfg::C, 1);
		int clusters = 0;
		e = cudaOccupancyMaxActiveClusters(&clusters, k_resident<LN, K, PCK, SOLO>, &cfg);
		if (e != cudaSuccess) { cudaGetLastError(); clusters = 0; }
		if (clusters > 0) ok.fetch_or(bit, std::memory_order_acq_rel);
		done.fetch_or(bit, std::memory_order_acq_rel);
		cfg.gridDim = dim3(Cfg::C, (unsigned)ncand);
	}
	const bool can = (ok.load(std::memory_order_acquire) & bit) != 0;
	if (fits) *fits = can;
	if (ncand == 0) return cudaSuccess;       // query and set-up only
	if (!can) return cudaErrorNotSupported;
	return cudaLaunchKernelEx(&cfg, k_resident<LN, K, PCK, SOLO>, J, c);
}

template <int LN, int K, int PCK>
cudaError_t resident_t(const ResJob & J, const TConst & c, cudaStream_t s, int ncand, bool * fits)
{
	if constexpr (LN >= 11)
	{
		if (ncand == 0)
		{
			// both set up before any capture
			const cudaError_t e = resident_v<LN, K, PCK, true>(J, c, s, 0, fits);
			if (e != cudaSuccess || (fits && !*fits)) return e;
		}
		if (ncand == 1) return resident_v<LN, K, PCK, true>(J, c, s, ncand, fits);
	}
	return resident_v<LN, K, PCK, false>(J, c, s, ncand, fits);
}

template <int K, int PCK>
cudaError_t resident_k(const ResJob & J, const TConst & c, cudaStream_t s, int ncand, bool * fits)
{
	switch (c.ln)
	{
	case 6: return resident_t<6, K, PCK>(J, c, s, ncand, fits);
	case 7: return resident_t<7, K, PCK>(J, c, s, ncand, fits);
	case 8: return resident_t<8, K, PCK>(J, c, s, ncand, fits);
	case 9: return resident_t<9, K, PCK>(J, c, s, ncand, fits);
	case 10: return resident_t<10, K, PCK>(J, c, s, ncand, fits);
	case 11: return resident_t<11, K, PCK>(J, c, s, ncand, fits);
	case 12: return resident_t<12, K, PCK>(J, c, s, ncand, fits);
	default: if (fits) *fits = false; return (ncand == 0) ? cudaSuccess : cudaErrorNotSupported;
	}
}

} // namespace
} // namespace ab
