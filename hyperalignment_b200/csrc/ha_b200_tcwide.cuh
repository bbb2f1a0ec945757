// ha_b200_tcwide.cuh -- the iteration's Gram and update products for searchlights too large for the
// chip-resident iteration (more than 256 vertices): the products of k_tc_gemm in the same order
// (identical bits) over 256-row tiles, one CTA per SM walking its tiles.
//
// With 128-row tiles, two CTAs per SM, 854 searchlights of 301-512 vertices took 574 us a Gram and 736 us an
// update launch.  Per tile of 256 columns and 31 slices (clock stamps): 4,000 cycles of prologue,
// 35,000 of products (60,000 for the update, whose A came through per-thread loads) and 12,000 of
// epilogue, where the tensor pipe needs 12,000: during the products both CTAs together read 43 B per
// cycle, all that an SM gets from L2.  Here
//   * a tile is 256 rows by up to 256 columns, two accumulators (all 512 tensor-memory columns): a third
//     less to read per product;
//   * the operands come by bulk copies of 2-4 KB, 32 of K a stage, except the update's K-major A, which four
//     warps load (512 contiguous bytes an instruction): as 64 bulk copies of 512 bytes a stage they took
//     4,300 cycles a stage, about 64 each whatever their size, and the launch 670 us.  Three stages of
//     64 KB run on into the next tile while the epilogue drains;
//   * the tiles' descriptors and the update's decisions are gathered once per launch;
//   * the epilogue moves the powers of two into the coefficients (exactly), as the resident form does.
// The same launches take 404 and 420 us (the 40 iterations of the solve 22.0 -> 15.6 ms); the products are
// 62% of a launch's cycles, the epilogue, which needs both accumulators, 28%.
#pragma once

#include "ha_b200_tcres.cuh"

namespace hab200 {

// warps 0-7 epilogue, 8 producer, 9 products; the update's loaders of A, 10-13
template <int PHASE>
constexpr int kTcWThreads = PHASE == kTcPhaseUpdate ? 448 : 320;
constexpr int kTcWStages = 3;
constexpr uint32_t kTcWPlane = 256 * 32 * 2;          // bytes of one operand plane of a stage
constexpr uint32_t kTcWStage = 4 * kTcWPlane;         // A hi, A mid, B hi, B mid
constexpr int kTcWMaxTiles = 256;                     // tiles per CTA (the grid grows to keep within it)
constexpr int kTcWSmem = kTcWStages * (int)kTcWStage + kTcWMaxTiles * (int)sizeof(TcIterTile);

// The tiles of one searchlight (work index w, np > 256): 256-row blocks times two column halves.
template <typename F>
inline void tcw_tiles(int w, int np, const F &put) {
	const int h0 = (np / 2 + 15) & ~15;
	for (int t = 0; t * 256 < np; t++) {
		put(TcTile{w, t, 0, h0});
		put(TcTile{w, t, h0, np - h0});
	}
}

// Epilogue of one 128-row tile (rows 128 t128 + 32 q ..): the accumulator holds 2^24 times the product.
template <int PHASE>
__device__ __forceinline__ void tcw_epilogue(const TcArgs &a, const TcIterTile &d, int t128, int q, int lane,
                                             uint32_t trow) {
	const int n = d.n, np = d.np, npg = np >> 3, n0 = d.n0, N = d.nn;
	const int row = 128 * t128 + 32 * q + lane;
	const int64_t pe = (int64_t)np * np;
	const bool fin = PHASE == kTcPhaseUpdate && d.fin;
	const float k3 = PHASE == kTcPhaseGram ? a.c3 * (1.f / 4096.f) : 1.f / 4096.f, k1 = a.c1 * 4096.f;
	__nv_bfloat16 *out = PHASE == kTcPhaseGram ? a.Pp + d.pofs : a.Xw + d.xofs;
	float res = 0.f;
	for (int cb = 0; cb < N; cb += 64) {
		// 64 columns per tensor-memory load (inside the 256-column accumulator; columns past N unused)
		float vv[64];
		tmem_ld64(trow + (uint32_t)cb, vv);
		const int dq = row - n0 - cb;  // the diagonal's place in these columns
		const bool diag = PHASE == kTcPhaseGram && __any_sync(0xffffffffu, dq >= 0 && dq < 64);
		if (row < np) {
#pragma unroll
			for (int sb = 0; sb < 4; sb++) {
				const int c0 = cb + 16 * sb;
				if (c0 >= N) break;
				float *v = vv + 16 * sb;
				if (fin) {
					if (row < n) {
						float *T = a.T + d.tofs;
#pragma unroll
						for (int k = 0; k < 16; k++) {
							const int col = n0 + c0 + k;
							if (col < n) T[a.t_rowmajor ? (int64_t)row * n + col : (int64_t)col * n + row] = v[k] * kTcAccUnscale;
						}
					}
					continue;
				}
				if (diag) {
#pragma unroll
					for (int k = 0; k < 16; k++) {
						// rows and columns past n are exactly zero and count nothing
						const float e = row < n && 16 * sb + k == dq ? v[k] - 16777216.f : v[k];
						res = fmaf(e, e, res);
						v[k] = fmaf(v[k], k3, 16 * sb + k == dq ? k1 : 0.f);
					}
				} else {
#pragma unroll
					for (int k = 0; k < 16; k++) {
						if (PHASE == kTcPhaseGram) res = fmaf(v[k], v[k], res);
						v[k] *= k3;
					}
				}
				uint32_t hi[8], mid[8];
				tcres_split16(v, hi, mid);
				const int64_t o = ((int64_t)(row >> 3) * npg + ((n0 + c0) >> 3)) * 64 + (row & 7) * 8;
				*reinterpret_cast<uint4 *>(out + o) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
				*reinterpret_cast<uint4 *>(out + o + 64) = make_uint4(hi[4], hi[5], hi[6], hi[7]);
				*reinterpret_cast<uint4 *>(out + pe + o) = make_uint4(mid[0], mid[1], mid[2], mid[3]);
				*reinterpret_cast<uint4 *>(out + pe + o + 64) = make_uint4(mid[4], mid[5], mid[6], mid[7]);
			}
		}
		__syncwarp();
	}
	if (PHASE == kTcPhaseGram) {
		res = warp_sum(res * 3.552713678800501e-15f);  // 2^-48
		if (lane == 0) a.res_part[(int64_t)d.slot * kTcResSlots + (2 * t128 + (n0 > 0 ? 1 : 0)) * 4 + q] = res;
	}
}

template <int PHASE>
__global__ void __launch_bounds__(kTcWThreads<PHASE>, 1) k_tc_wide(const TcArgs a, int ntiles) {
	static_assert(PHASE != kTcPhaseXcov, "the cross-covariance has its own kernel");
	extern __shared__ __align__(128) unsigned char tw_smem[];
	__shared__ uint64_t s_full[kTcWStages], s_empty[kTcWStages], s_accf, s_acce, s_done;
	__shared__ uint32_t s_tmem;
	__shared__ int s_fail;
	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
	// tiles dealt in snake order, which balances a largest-first list better than round-robin
	const int G = (int)gridDim.x, B = (int)blockIdx.x;
	auto tile_of = [&](int e) { return e * G + ((e & 1) ? G - 1 - B : B); };
	int mine = ntiles / G;
	if (mine * G < ntiles && tile_of(mine) < ntiles) mine++;
	TcIterTile *tlist = reinterpret_cast<TcIterTile *>(tw_smem + kTcWStages * kTcWStage);
	const uint32_t smem0 = smem_u32(tw_smem);
	if (tid == 0) {
		for (int i = 0; i < kTcWStages; i++) {
			mbar_init(&s_full[i], PHASE == kTcPhaseUpdate ? 129 : 1);
			mbar_init(&s_empty[i], 1);
		}
		mbar_init(&s_accf, 1);
		mbar_init(&s_acce, 8);
		mbar_init(&s_done, 1);
		s_fail = (mine > kTcWMaxTiles || (PHASE == kTcPhaseUpdate && a.Xw == nullptr)) ? 1 : 0;
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	if (warp == 0) tmem_alloc(&s_tmem, 512);
	if (mine <= kTcWMaxTiles)
		for (int e = tid; e < mine; e += kTcWThreads<PHASE>) {
			const TcTile tl = a.tiles[tile_of(e)];
			const TcWork w = a.work[tl.w];
			const TcState st = a.st_in[w.slot];
			TcIterTile d;
			d.slot = w.slot; d.n = w.n; d.np = w.np; d.t = tl.t; d.n0 = tl.n0; d.nn = tl.nn;
			d.skip = st.done ? 1 : 0;
			d.fin = 0;
			d.xofs = w.xofs; d.pofs = w.pofs; d.tofs = w.tofs;
			if (PHASE == kTcPhaseUpdate) {
				TcState o = st;
				if (!st.done) d.fin = tc_update_decision(a, w, st, &o) ? 1 : 0;
				if (tl.t == 0 && tl.n0 == 0) a.st_out[w.slot] = o;
			}
			tlist[e] = d;
		}
	tc_fence_before();
	__syncthreads();
	tc_fence_after();
	const uint32_t tmem = s_tmem;
	volatile int *vfail = &s_fail;
	const bool failed0 = *vfail != 0;

	if (warp == 8 && !failed0) {
		uint32_t g = 0;  // stages filled
		bool ok = true;
		for (int e = 0; e < mine && ok; e++) {
			const TcIterTile d = tlist[e];
			if (d.skip) continue;
			const int np = d.np, npg = np >> 3, N = d.nn, nk = np >> 4, gA = min(32, npg - 32 * d.t);
			const int64_t pe = (int64_t)np * np;
			const __nv_bfloat16 *X = a.Xp + d.xofs;
			const __nv_bfloat16 *Bs = ((PHASE == kTcPhaseGram) ? X : (const __nv_bfloat16 *)(a.Pp + d.pofs)) + (d.n0 >> 3) * 64;
			for (int ks = 0; ks < nk; ks += 2, g++) {
				const int s = (int)(g % kTcWStages), kn = min(2, nk - ks);
				int go = 1;
				if (lane == 0) {
					if (*vfail || (g >= kTcWStages && !mbar_wait(&s_empty[s], (g / kTcWStages - 1) & 1u))) {
						*vfail = 1;
						go = 0;
					}
					if (go) mbar_expect_tx(&s_full[s], (uint32_t)kn * ((PHASE == kTcPhaseGram ? 512u * (uint32_t)gA : 0u) + 64u * (uint32_t)N));
				}
				if (!__shfl_sync(0xffffffffu, go, 0)) {
					ok = false;
					break;
				}
				const uint32_t st = smem0 + (uint32_t)s * kTcWStage;
				const int p = (lane >> 2) & 1, o = lane & 3;  // plane and 8-sample part of K
				if (lane < 8 && o < 2 * kn)
					bulk_g2s(st + (2 + p) * kTcWPlane + (uint32_t)(o * 16 * N), Bs + p * pe + (int64_t)(2 * ks + o) * npg * 64, 16u * N, &s_full[s]);
				// the Gram's A, columns of X: one piece per part
				if (PHASE == kTcPhaseGram && lane >= 8 && lane < 16 && o < 2 * kn)
					bulk_g2s(st + p * kTcWPlane + o * 4096u, X + p * pe + ((int64_t)(2 * ks + o) * npg + 32 * d.t) * 64, 128u * gA, &s_full[s]);
			}
		}
		// every copy issued has landed before the CTA may leave (after a failure the bounded waits run out)
		if (lane == 0)
			for (uint32_t h = g > (uint32_t)kTcWStages ? g - kTcWStages : 0u; h < g; h++)
				if (!mbar_wait(&s_full[h % kTcWStages], (h / kTcWStages) & 1u)) *vfail = 1;
		__syncwarp();
	}
	if (PHASE == kTcPhaseUpdate && warp >= 10 && !failed0) {
		// rows of X: chunk c of a plane (16 bytes) is row c % 8 of core (c / 32, (c / 8) % 4), the same order in
		// memory and in the stage; a warp's instruction is four cores along K
		uint32_t g = 0;
		bool ok = true;
		const int lt = tid - 320, k8 = (lt >> 3) & 3;
		for (int e = 0; e < mine && ok; e++) {
			const TcIterTile d = tlist[e];
			if (d.skip) continue;
			const int np = d.np, npg = np >> 3, nk = np >> 4, gA = min(32, npg - 32 * d.t) - (lt >> 5);
			const int64_t pe = (int64_t)np * np, gs = (int64_t)npg * 256;  // four groups of eight rows
			const __nv_bfloat16 *src = a.Xp + d.xofs + ((int64_t)(32 * d.t + (lt >> 5)) * npg + k8) * 64 + 8 * (lt & 7);
			for (int ks = 0; ks < nk; ks += 2, g++) {
				const int s = (int)(g % kTcWStages);
				int go = 1;
				if (lane == 0 && (*vfail || (g >= kTcWStages && !mbar_wait(&s_empty[s], (g / kTcWStages - 1) & 1u)))) {
					*vfail = 1;
					go = 0;
				}
				if (!__shfl_sync(0xffffffffu, go, 0)) {
					ok = false;
					break;
				}
				const uint32_t dst = smem0 + (uint32_t)s * kTcWStage + 16u * (uint32_t)lt;
				const __nv_bfloat16 *at = src + (int64_t)ks * 128;
				if (2 * ks + k8 < npg)
#pragma unroll
					for (int p = 0; p < 2; p++)
#pragma unroll
						for (int j = 0; j < 8; j++)
							if (4 * j < gA) cp_async16(dst + p * kTcWPlane + 2048u * j, at + p * pe + j * gs, 16u);
				cp_async_arrive_noinc(&s_full[s]);
			}
		}
		cp_async_wait_all();
	}
	if (warp == 9 && !failed0) {
		if (lane == 0) {
			uint32_t g = 0, j = 0;  // stages consumed, tiles computed
			const uint32_t lba = PHASE == kTcPhaseGram ? 4096 : 128, sba = PHASE == kTcPhaseGram ? 128 : 512;
			const uint32_t ta = PHASE == kTcPhaseGram ? 2048 : 8192;  // the second 128 rows of A
			for (int e = 0; e < mine && !*vfail; e++) {
				const TcIterTile d = tlist[e];
				if (d.skip) continue;
				const int nk = d.np >> 4, N = d.nn, two = d.np - 256 * d.t > 128;
				const uint32_t id = mma_idesc(128, N, PHASE == kTcPhaseGram ? 1 : 0, 1, true);
				if (j >= 1 && !mbar_wait(&s_acce, (j - 1) & 1u)) {
					*vfail = 1;
					break;
				}
				tc_fence_after();
				for (int ks = 0; ks < nk; ks += 2, g++) {
					const int s = (int)(g % kTcWStages), kn = min(2, nk - ks);
					if (!mbar_wait(&s_full[s], (g / kTcWStages) & 1u)) {
						*vfail = 1;
						break;
					}
					if (PHASE == kTcPhaseUpdate) fence_proxy_async_smem();  // the loaders' writes, seen through the barrier, to the products
					tc_fence_after();
					const uint32_t st = smem0 + (uint32_t)s * kTcWStage;
					for (int sl = 0; sl < kn; sl++)
						for (int t = 0; t <= two; t++)
#pragma unroll
							for (int q = 0; q < 3; q++)  // mid*hi, hi*mid, hi*hi
								mma_bf16(tmem + 256u * t,
								         smem_desc(st + (q == 0 ? kTcWPlane : 0u) + 2u * sl * lba + ta * t, lba, sba),
								         smem_desc(st + (q == 1 ? 3u : 2u) * kTcWPlane + (uint32_t)(sl * 32 * N), 16u * N, 128), id,
								         (ks > 0 || sl > 0 || q > 0) ? 1u : 0u);
					mma_commit(&s_empty[s]);
				}
				if (*vfail) break;
				mma_commit(&s_accf);
				j++;
			}
			mma_commit(&s_done);  // completes once every product issued has
			if (!mbar_wait(&s_done, 0)) *vfail = 1;
		}
		__syncwarp();
	}
	if (warp < 8 && !failed0) {
		uint32_t j = 0;
		const int q = warp & 3, t = warp >> 2;
		for (int e = 0; e < mine; e++) {
			const TcIterTile d = tlist[e];
			if (d.skip) continue;
			int ok = 1;
			if (lane == 0) ok = mbar_wait_idle(&s_accf, j & 1u) && !*vfail ? 1 : 0;
			if (!__shfl_sync(0xffffffffu, ok, 0)) {
				*vfail = 1;
				break;
			}
			tc_fence_after();
			if (256 * d.t + 128 * t < d.np)
				tcw_epilogue<PHASE>(a, d, 2 * d.t + t, q, lane, tmem + 256u * t + ((uint32_t)(32 * q) << 16));
			tc_fence_before();
			__syncwarp();
			if (lane == 0) mbar_arrive(&s_acce);
			j++;
		}
	}
	__syncwarp();
	tc_fence_before();
	__syncthreads();
	if (tid == 0 && s_fail) atomicOr(a.err, 1);
	if (warp == 0) tmem_dealloc(tmem, 512);
}

}  // namespace hab200
