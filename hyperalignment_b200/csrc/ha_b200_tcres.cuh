// ha_b200_tcres.cuh -- the Newton-Schulz polar iteration of ha_b200_tc.cuh with a searchlight's
// iterate resident on the chip: the same products in the same order (identical bits), one launch for
// the whole iteration.
//
// The per-phase kernels stream every searchlight's planes through memory twice per iteration (20 np^2
// bytes) and drain a 13-slice pipeline per tile: measured 20-24% of the tensor pipe and 30-40% of the
// memory bandwidth.  Here one CTA (np <= 128) or a pair of CTAs (np <= 256, cta_group::2) keeps
//   * one panel in shared memory, the columns [h c, h c + h) of X, then of P, then of the next X
//     (c: the CTA's rank, h = N / CTAs): core matrices as in HBM, so the panel is an MN-major operand.
//     It is A and B of the Gram product (rows and columns of G are both columns of X), and B of the
//     update; P overwrites X and the next X overwrites P, each after the product that read it;
//   * the CTA's rows of X in tensor memory as the K-major A operand of the update;
//   * the accumulator beside it (np + np tensor-memory columns).
// CTA c computes the rows [h c, h c + h) of both products (an M = 128 tile a CTA; what it computes for
// rows past h is ignored) and sends each row's columns to the CTA that holds them.  The warps issue,
// wait, drain the accumulator (lane = row) and refill the panel together; a barrier of the cluster
// stands before each product.  They form G groups of four (a group covers the 128 lanes): the rows'
// residuals are sums in column order, so one group takes them while the others split 16-column blocks,
// those of the other CTA's panel first.  Every mbarrier wait is bounded; a failed one raises a flag in
// both CTAs, which leave together after the next barrier.
#pragma once

#include "ha_b200_tc.cuh"

namespace hab200 {

constexpr int kTcResMaxNp = 256;

struct TcResArgs {
	const TcWork *work;
	const int32_t *order;     // work indices of the launch
	const __nv_bfloat16 *X0;  // iterate planes (TcWork::xofs)
	float *T;                 // T scratch (TcWork::tofs)
	int t_rowmajor;
	const TcState *st_in;
	TcState *st_out;
	const float *c1, *c3;     // schedule, maxit entries
	const int32_t *plain;
	int maxit;
	float tol_stop;
	int *err;
};

// Panel of one CTA: kp rows (np), h columns, two planes, and room for the rows of A past h that the
// last K slice reads.
__host__ __device__ __forceinline__ int tcres_n(int np, int cl) { return cl == 2 ? (np + 31) & ~31 : np; }
__host__ __device__ __forceinline__ size_t tcres_smem(int np, int cl) {
	return (size_t)np * (tcres_n(np, cl) / cl) * 4 + 16 * 128;
}

template <int CL>
__device__ __forceinline__ uint32_t tcres_rank() {
	uint32_t r = 0;
	if (CL == 2) asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
	return r;
}
__device__ __forceinline__ uint32_t tcres_mapa(uint32_t addr, uint32_t rank) {
	uint32_t r;
	asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
	return r;
}
__device__ __forceinline__ void tcres_st16(uint32_t addr, uint4 v, bool remote) {
	if (remote)
		asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
		             : "memory");
	else
		asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
		             : "memory");
}
__device__ __forceinline__ void tcres_st4(uint32_t addr, uint32_t v) {
	asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

template <int CL>
__device__ __forceinline__ void tcres_barrier() {
	if (CL == 2) {
		asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
		asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
	} else {
		__syncthreads();
	}
}

// Everything this thread wrote (shared memory of either CTA, tensor memory) is visible to the products
// issued after the barrier, and its tensor-memory reads precede them.
template <int CL>
__device__ __forceinline__ void tcres_ready() {
	asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
	asm volatile("fence.proxy.async;" ::: "memory");
	tc_fence_before();
	tcres_barrier<CL>();
	tc_fence_after();
}

template <int CL>
__device__ __forceinline__ void tcres_alloc(uint32_t *dst, uint32_t ncols) {
	if (CL == 2) {
		asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst)), "r"(ncols) : "memory");
		asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
	} else {
		tmem_alloc(dst, ncols);
	}
}
template <int CL>
__device__ __forceinline__ void tcres_dealloc(uint32_t base, uint32_t ncols) {
	if (CL == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(ncols) : "memory");
	else tmem_dealloc(base, ncols);
}

// A in shared memory (desc) or tensor memory (address).
template <int CL>
__device__ __forceinline__ void tcres_mma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
	if (CL == 2)
		asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
		             "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
		             : "memory");
	else
		mma_bf16(d, a, b, idesc, accumulate);
}
template <int CL>
__device__ __forceinline__ void tcres_mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
	if (CL == 2)
		asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
		             "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate)
		             : "memory");
	else
		asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
		             "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate)
		             : "memory");
}
// Arrive on `bar` of every CTA of the cluster once the products issued so far have completed.
template <int CL>
__device__ __forceinline__ void tcres_commit(uint64_t *bar) {
	if (CL == 2)
		asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
		             "h"((uint16_t)3)
		             : "memory");
	else
		mma_commit(bar);
}

// 8 consecutive tensor-memory columns of this warp's 32 lanes.
__device__ __forceinline__ void tcres_st8(uint32_t taddr, const uint32_t *r) {
	asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]),
	             "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
	             : "memory");
}

// 16 values x 2^12 -> their FP16 hi and mid parts, two to a word (the split of store_split8h).
__device__ __forceinline__ void tcres_split16(const float *a, uint32_t *hi, uint32_t *mid) {
#pragma unroll
	for (int i = 0; i < 8; i++) {
		const __half2 h = __floats2half2_rn(a[2 * i], a[2 * i + 1]);
		const __half2 m = __floats2half2_rn(a[2 * i] - __low2float(h), a[2 * i + 1] - __high2float(h));
		hi[i] = *reinterpret_cast<const uint32_t *>(&h);
		mid[i] = *reinterpret_cast<const uint32_t *>(&m);
	}
}

template <int CL, int G>
__global__ void __launch_bounds__(128 * G) k_tc_resident(const TcResArgs a) {
	extern __shared__ __align__(128) unsigned char tr_smem[];
	__shared__ __align__(8) uint64_t s_bar;
	__shared__ uint32_t s_tmem;
	__shared__ int s_fail;
	__shared__ float s_rr[kTcResMaxNp];  // squared residual of every row (of both CTAs)
	__shared__ int s_fin;
	constexpr int kThreads = 128 * G;
	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, quarter = warp & 3, group = warp >> 2;
	const uint32_t rank = tcres_rank<CL>();
	const TcWork w = a.work[a.order[blockIdx.x / CL]];
	const int n = w.n, kp = w.np, N = tcres_n(kp, CL), h = N / CL, gh = h >> 3, npg = kp >> 3, nk = kp >> 4;
	const uint32_t plane = (uint32_t)kp * h * 2;  // bytes of a panel plane
	const uint32_t own = smem_u32(tr_smem);
	uint32_t panel[CL];  // each CTA's panel as this CTA addresses it
#pragma unroll
	for (int c = 0; c < CL; c++) panel[c] = c == (int)rank ? own : tcres_mapa(own, c);
	const int lrow = 32 * quarter + lane, row = (int)rank * h + lrow;  // row of X; the accumulator's lane
	const bool mine = lrow < h && row < kp;
	// accumulator in columns [0, N), the rows of X behind it: hi words, then mid words
	const uint32_t acol = (uint32_t)((N + 31) & ~31);
	uint32_t ncols = 32;
	while (ncols < acol + (uint32_t)kp) ncols <<= 1;

	if (tid == 0) {
		mbar_init(&s_bar, 1);
		s_fail = 0;
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	for (int i = tid; i < kTcResMaxNp; i += kThreads) s_rr[i] = 0.f;
	if (warp == 0) tcres_alloc<CL>(&s_tmem, ncols);
	tc_fence_before();
	tcres_barrier<CL>();
	tc_fence_after();
	const uint32_t tmem = s_tmem;
	const uint32_t trow = tmem + ((uint32_t)(32 * quarter) << 16);
	const uint32_t arow = trow + acol;

	// X_0: the panel's cores as they lie in HBM, and the CTA's rows into tensor memory
	{
		const uint4 *src = reinterpret_cast<const uint4 *>(a.X0 + w.xofs);
		const int c0 = (int)rank * gh, cn = min(gh, npg - c0);  // 8-column groups of the panel that exist
		const int per = npg * cn * 8;                          // 16-byte rows of a plane
#pragma unroll 8
		for (int e = tid; e < 2 * per; e += kThreads) {
			const int p = e >= per ? 1 : 0, f = e - p * per, r = f & 7, core = f >> 3, rg = core / cn, cg = core - rg * cn;
			const uint4 v = src[(int64_t)p * npg * npg * 8 + ((int64_t)rg * npg + c0 + cg) * 8 + r];
			tcres_st16(own + p * plane + (uint32_t)((rg * gh + cg) * 128 + r * 16), v, false);
		}
		const int rs = min(row, kp - 1);
		for (int c = 2 * group; c < npg; c += 2 * G) {  // 16 columns: 8 words a plane
#pragma unroll
			for (int p = 0; p < 2; p++) {
				const uint4 *q = src + (int64_t)p * npg * npg * 8 + ((int64_t)(rs >> 3) * npg + c) * 8 + (rs & 7);
				const uint4 x = q[0], y = q[8];
				const uint32_t wd[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
				tcres_st8(arow + p * (kp >> 1) + 4 * c, wd);
			}
		}
	}

	const uint32_t id_gram = mma_idesc(128 * CL, N, 1, 1, true), id_upd = mma_idesc(128 * CL, N, 0, 1, true);
	const uint32_t kstride = (uint32_t)gh * 128;  // bytes between 8-row groups of the panel
	TcState st = a.st_in[w.slot];
	uint32_t phase = 0;
	bool finished = false;
	// one warp polls and the others stand at the barrier: polling warps take the issue slots of the one
	// that issues the products and of the one that decides
	auto wait_products = [&]() {
		if (warp == 1 && !mbar_wait(&s_bar, phase)) {
#pragma unroll
			for (int c = 0; c < CL; c++) tcres_st4(CL == 2 ? tcres_mapa(smem_u32(&s_fail), c) : smem_u32(&s_fail), 1u);
		}
		phase ^= 1u;
		__syncthreads();
		tc_fence_after();
	};
	// the 16-column blocks, those of the other CTA's panel first
	const int first = CL == 2 && rank == 0 ? h >> 4 : 0;
	auto block_at = [&](int i) {
		const int b = i + first;
		return 16 * (b < nk ? b : b - nk);
	};
	// 16 columns of this thread's row into the panel that holds them
	auto put = [&](int c0, const uint32_t *hi, const uint32_t *mid) {
		if (!mine) return;
		const int c = CL == 2 && c0 >= h ? 1 : 0;
		const bool remote = CL == 2 && c != (int)rank;
		const uint32_t at = (CL == 2 && c ? panel[CL - 1] : panel[0]) +
		                    (uint32_t)(((row >> 3) * gh + ((c0 - c * h) >> 3)) * 128 + (row & 7) * 16);
		tcres_st16(at, make_uint4(hi[0], hi[1], hi[2], hi[3]), remote);
		tcres_st16(at + 128, make_uint4(hi[4], hi[5], hi[6], hi[7]), remote);
		tcres_st16(at + plane, make_uint4(mid[0], mid[1], mid[2], mid[3]), remote);
		tcres_st16(at + plane + 128, make_uint4(mid[4], mid[5], mid[6], mid[7]), remote);
	};
	for (int k = 0; k < a.maxit; k++) {
		const float c1 = a.c1[k], c3 = a.c3[k];
		const bool plain = a.plain[k] != 0;
		// G = X^T X
		tcres_ready<CL>();
		if (*(volatile int *)&s_fail) break;
		if (rank == 0 && tid == 0) {
			asm volatile("fence.proxy.async;" ::: "memory");
			for (int ks = 0; ks < nk; ks++)
#pragma unroll
				for (int q = 0; q < 3; q++) {  // mid*hi, hi*mid, hi*hi
					const uint32_t at = own + (uint32_t)(2 * ks) * kstride;
					tcres_mma_ss<CL>(tmem, smem_desc(at + (q == 0 ? plane : 0u), kstride, 128),
					                 smem_desc(at + (q == 1 ? plane : 0u), kstride, 128), id_gram, (ks > 0 || q > 0) ? 1u : 0u);
				}
			tcres_commit<CL>(&s_bar);
		}
		wait_products();
		// P = c1 I + c3 G over the panels, the rows' residuals.  The accumulator holds 2^24 G; what
		// follows is the per-phase kernels' arithmetic with its powers of two moved (exactly).
		if (group == 0) {
			float res = 0.f;
			for (int cb = 0; cb < kp; cb += 64) {
				float v[64];
				tmem_ld64(trow + (uint32_t)cb, v);
				const int dq = row < n ? row - cb : -1;  // the diagonal's place in these columns
				const bool diag = __any_sync(0xffffffffu, dq >= 0 && dq < 64);
#pragma unroll
				for (int s = 0; s < 4; s++) {
					if (cb + 16 * s >= kp) break;
#pragma unroll
					for (int q = 16 * s; q < 16 * s + 16; q++) {
						const float d = diag && q == dq ? v[q] - 16777216.f : v[q];
						res = fmaf(d, d, res);
					}
				}
			}
			if (mine) {
				const uint32_t rv = __float_as_uint(res * 3.552713678800501e-15f);  // 2^-48
#pragma unroll
				for (int c = 0; c < CL; c++) {
					const uint32_t at = smem_u32(&s_rr[row]);
					tcres_st4(CL == 2 ? tcres_mapa(at, c) : at, rv);
				}
			}
		} else {
			const float k3 = c3 * (1.f / 4096.f), k1 = c1 * 4096.f;
			for (int i = group - 1; i < nk; i += G - 1) {
				const int c0 = block_at(i), dq = row - c0;
				float v[16];
				tmem_ld16(trow + (uint32_t)c0, v);
				if (__any_sync(0xffffffffu, dq >= 0 && dq < 16)) {
#pragma unroll
					for (int q = 0; q < 16; q++) v[q] = fmaf(v[q], k3, q == dq ? k1 : 0.f);
				} else {
#pragma unroll
					for (int q = 0; q < 16; q++) v[q] *= k3;
				}
				uint32_t hi[8], mid[8];
				tcres_split16(v, hi, mid);
				put(c0, hi, mid);
			}
		}
		// X <- X P
		tcres_ready<CL>();
		if (*(volatile int *)&s_fail) break;
		if (rank == 0 && tid == 0) {
			asm volatile("fence.proxy.async;" ::: "memory");
			for (int ks = 0; ks < nk; ks++)
#pragma unroll
				for (int q = 0; q < 3; q++)
					tcres_mma_ts<CL>(tmem, tmem + acol + (q == 0 ? (uint32_t)(kp >> 1) : 0u) + 8u * ks,
					                 smem_desc(own + (uint32_t)(2 * ks) * kstride + (q == 1 ? plane : 0u), kstride, 128), id_upd,
					                 (ks > 0 || q > 0) ? 1u : 0u);
			tcres_commit<CL>(&s_bar);
		}
		// the decision, while the products run, by a warp that issues none: the partial sums of the
		// per-phase kernels (32 rows each), in their order
		if (warp == 4) {
			float part[kTcResMaxNp / 32];
#pragma unroll
			for (int g = 0; g < kTcResMaxNp / 32; g++) part[g] = s_rr[32 * g + lane];
#pragma unroll
			for (int o = 16; o > 0; o >>= 1)
#pragma unroll
				for (int g = 0; g < kTcResMaxNp / 32; g++) part[g] += __shfl_xor_sync(0xffffffffu, part[g], o);
			double ss = 0.0;
#pragma unroll
			for (int g = 0; g < kTcResMaxNp / 32; g++) ss += (double)part[g];  // rows past np hold zeros
			const double resd = sqrt(ss / (double)n);
			const float r32 = (float)resd;
			const bool conv = plain && r32 < a.tol_stop;
			const bool stalled = !conv && plain && st.plain && fabs(resd - (double)st.res) <= 5e-7 * resd;
			const bool fin = conv || stalled || k == a.maxit - 1;
			st.iters++;
			st.res = r32;
			st.conv = conv ? 1 : 0;
			st.stalled = stalled ? 1 : 0;
			st.done = fin ? 1 : 0;
			st.plain = plain ? 1 : 0;
			if (lane == 0) s_fin = fin ? 1 : 0;
		}
		wait_products();
		if (s_fin) {
			float *T = a.T + w.tofs;
			for (int c0 = 16 * group; c0 < n; c0 += 16 * G) {
				float v[16];
				tmem_ld16(trow + (uint32_t)c0, v);
				if (lrow < h && row < n)
#pragma unroll
					for (int q = 0; q < 16; q++) {
						const int col = c0 + q;
						if (col < n) T[a.t_rowmajor ? (int64_t)row * n + col : (int64_t)col * n + row] = v[q] * kTcAccUnscale;
					}
			}
			finished = true;
			break;
		}
		for (int i = group; i < nk; i += G) {
			const int c0 = block_at(i);
			float v[16];
			tmem_ld16(trow + (uint32_t)c0, v);
#pragma unroll
			for (int q = 0; q < 16; q++) v[q] *= 1.f / 4096.f;
			uint32_t hi[8], mid[8];
			tcres_split16(v, hi, mid);
			put(c0, hi, mid);
			tcres_st8(arow + (uint32_t)(c0 >> 1), hi);
			tcres_st8(arow + (uint32_t)((kp + c0) >> 1), mid);
		}
	}
	if (warp == 4 && lane == 0) {
		if (!finished || *(volatile int *)&s_fail) atomicOr(a.err, 1);
		if (rank == 0) a.st_out[w.slot] = st;
	}
	tcres_ready<CL>();  // neither CTA leaves while the other may still reach its shared or tensor memory
	if (warp == 0) tcres_dealloc<CL>(tmem, ncols);
}

}  // namespace hab200
