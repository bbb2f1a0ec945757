// ha_b200_tcxcov.cuh -- the cross-covariance A = X_sl^T Y_sl of the tensor-core solver
// (csrc/ha_searchlight.c:581-582): split BF16, three parts and six products per K slice of 16, FP32
// accumulation in tensor memory.
//
// The operands are gathered rows of time series, and the requests to L2 bound it.  With one 128-row tile
// a CTA, 16-byte pieces of 16 different rows per warp instruction and the columns' rows read again for
// every row tile, 9,675 searchlights of 90-170 vertices and 1,818 samples took 10.7 ms.  Here a CTA
// computes up to 256 rows (two accumulators) from one copy of the columns' rows and a stage holds 32
// samples (64 bytes) of each: 7.2 ms while the pieces of a row were scattered in shared memory (one
// request per 32-byte sector, counted), 5.1 ms with them in one swizzled 64-byte line.  10,242
// searchlights of 100-300 vertices and 400 samples: 5.6 -> 3.0 ms; 854 of 301-512 and 1,000: 3.5 -> 1.5 ms.
#pragma once

#include "ha_b200_tc.cuh"

namespace hab200 {

constexpr int kTcXThreads = 288;  // eight producer (then epilogue) warps, one that issues the products
constexpr int kTcXProducers = 256;
constexpr int kTcXK = 32;         // samples per stage
constexpr int kTcXRows = 256;     // rows and columns per CTA at most

struct TcXArgs {
	const TcWork *work;
	const TcTile *tiles;  // t: 256-row block, columns [n0, n0 + nn)
	const __nv_bfloat16 *Xb;
	const __nv_bfloat16 *Yb;
	int64_t vplane;       // elements per vertex-major plane (nv * ntp)
	int ntp;              // samples per row, a multiple of kTcXK (zero padded, so a stage stays in its row)
	const int32_t *sl_idx;
	float *A32;
	int smem_bytes;
	int *err;
};

// Operand of a stage: a plane is rows of 64 bytes (32 samples) in the 64-byte swizzle: 16-byte piece c of
// row r at 64 r + 16 (c ^ ((r / 2) % 4)), planes 1 KB aligned.  The pieces of a row then go to one 64-byte
// line of shared memory, without which every 32-byte sector was a request of its own; eight lanes' pieces
// (two rows) fall into different banks.  A 128-row product reads rows past the operand's last (their results
// are not stored): at most 8 KB from a row plane's start, inside the allocation.
__host__ __device__ __forceinline__ int tcx_stage(int rows, int cols) { return 192 * (rows + cols); }
constexpr int kTcXAlign = 1024;
// Dynamic shared memory of the two size classes: two CTAs per SM where two stages fit half the shared
// memory and one accumulator of at most 256 columns is used, else one CTA per SM.
constexpr int kTcXSmem[2] = {110 * 1024, 224 * 1024};
inline int tcx_class(int rows, int cols) {
	return rows > 128 || 2 * tcx_stage(rows, cols) > kTcXSmem[0] - kTcXAlign ? 1 : 0;
}

// Shared-memory matrix descriptor, 64-byte swizzle, K-major: 512 bytes between 8-row groups.
__device__ __forceinline__ uint64_t smem_desc_sw64(uint32_t saddr) {
	return smem_desc(saddr, 16, 512) | ((uint64_t)4 << 61);
}

// The tiles of one searchlight (work index w): 256-row blocks, and two column halves past 256.
template <typename F>
inline void tcx_tiles(int w, int np, const F &put) {
	const int h0 = np > kTcXRows ? ((np / 2 + 15) & ~15) : np;
	for (int t = 0; t * kTcXRows < np; t++) {
		const int rows = np - t * kTcXRows < kTcXRows ? np - t * kTcXRows : kTcXRows;
		put(tcx_class(rows, h0), TcTile{w, t, 0, h0});
		if (h0 < np) put(tcx_class(rows, np - h0), TcTile{w, t, h0, np - h0});
	}
}

__global__ void __launch_bounds__(kTcXThreads) k_tc_xcov(const TcXArgs a) {
	extern __shared__ __align__(128) unsigned char tx_smem[];
	__shared__ uint64_t s_full[kTcMaxStages], s_empty[kTcMaxStages], s_acc;
	__shared__ uint32_t s_tmem;
	__shared__ int s_fail;
	__shared__ int32_t s_row[kTcXRows], s_col[kTcXRows];  // vertices of the rows and columns, -1: none
	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
	const TcTile tl = a.tiles[blockIdx.x];
	const TcWork w = a.work[tl.w];
	const int n = w.n, np = w.np, r0 = kTcXRows * tl.t, rows = min(kTcXRows, np - r0), N = tl.nn, n0 = tl.n0;
	const int ntiles = (rows + 127) >> 7;
	const int pa = 64 * rows, pb = 64 * N, stage_bytes = tcx_stage(rows, N);
	const int S = min(kTcMaxStages, (a.smem_bytes - kTcXAlign) / stage_bytes);
	const int nst = a.ntp / kTcXK;
	const uint32_t acc1 = (uint32_t)((N + 31) & ~31);  // the second tile's accumulator column
	uint32_t ncols = 32;
	while (ncols < acc1 * (uint32_t)ntiles) ncols <<= 1;
	const uint32_t smem0 = (smem_u32(tx_smem) + kTcXAlign - 1) & ~(uint32_t)(kTcXAlign - 1);
	if (tid == 0) {
		for (int i = 0; i < kTcMaxStages; i++) {
			mbar_init(&s_full[i], kTcXProducers);
			mbar_init(&s_empty[i], 1);
		}
		mbar_init(&s_acc, 1);
		s_fail = S < 2 ? 1 : 0;
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	for (int i = tid; i < kTcXRows; i += kTcXThreads) {
		s_row[i] = i < rows && r0 + i < n ? a.sl_idx[w.sofs + r0 + i] : -1;
		s_col[i] = i < N && n0 + i < n ? a.sl_idx[w.sofs + n0 + i] : -1;
	}
	if (warp == 0) tmem_alloc(&s_tmem, ncols);
	tc_fence_before();
	__syncthreads();
	tc_fence_after();
	const uint32_t tmem = s_tmem;
	volatile int *vfail = &s_fail;
	if (!*vfail && warp < 8) {
		// producers: lane = (row pair, chunk); a warp instruction covers eight rows
		const int q = lane & 3, rl = 8 * warp + (lane >> 2);
		constexpr int kPer = kTcXRows / 64;
		int64_t ro[kPer], co[kPer];  // element offsets of this lane's pieces; none: the planes' start, 0 bytes
		uint32_t rb[kPer], cb[kPer];
#pragma unroll
		for (int i = 0; i < kPer; i++) {
			const int r = s_row[rl + 64 * i], c = s_col[rl + 64 * i];
			ro[i] = r >= 0 ? (int64_t)r * a.ntp + 8 * q : 0;
			co[i] = c >= 0 ? (int64_t)c * a.ntp + 8 * q : 0;
			rb[i] = r >= 0 ? 16u : 0u;
			cb[i] = c >= 0 ? 16u : 0u;
		}
		const uint32_t lo = (uint32_t)(64 * rl + 16 * (q ^ ((rl >> 1) & 3)));  // rows 64 apart share the swizzle
		for (int k = 0; k < nst; k++) {
			const int s = k % S;
			if (k >= S) {
				int ok = 1;
				if (lane == 0) ok = !*vfail && mbar_wait(&s_empty[s], (uint32_t)((k / S - 1) & 1)) ? 1 : 0;
				if (!__shfl_sync(0xffffffffu, ok, 0)) {
					*vfail = 1;
					break;
				}
			}
			const uint32_t st = smem0 + (uint32_t)(s * stage_bytes);
			const int t0 = k * kTcXK;
#pragma unroll
			for (int p = 0; p < 3; p++) {
				const __nv_bfloat16 *Xp = a.Xb + p * a.vplane + t0, *Yp = a.Yb + p * a.vplane + t0;
				const uint32_t da = st + (uint32_t)(p * pa) + lo, db = st + (uint32_t)(3 * pa + p * pb) + lo;
#pragma unroll
				for (int i = 0; i < kPer; i++) {
					const int r = rl + 64 * i;
					if (r < rows) cp_async16(da + 4096u * i, Xp + ro[i], rb[i]);
					if (r < N) cp_async16(db + 4096u * i, Yp + co[i], cb[i]);
				}
			}
			cp_async_arrive_noinc(&s_full[s]);
		}
		cp_async_wait_all();
	}
	if (!*vfail && warp == 8) {
		if (lane == 0) {
			const uint32_t id = mma_idesc(128, N, 0, 0, false);
			for (int k = 0; k < nst; k++) {
				const int s = k % S;
				if (!mbar_wait(&s_full[s], (uint32_t)((k / S) & 1))) {
					*vfail = 1;
					break;
				}
				fence_proxy_async_smem();
				tc_fence_after();
				const uint32_t st = smem0 + (uint32_t)(s * stage_bytes);
				for (int sl = 0; sl < kTcXK / 16; sl++)
					for (int t = 0; t < ntiles; t++) {
#pragma unroll
						for (int q = 0; q < 6; q++) {  // lo*hi, hi*lo, mid*mid, mid*hi, hi*mid, hi*hi
							const int xa = (q == 0) ? 2 : (q == 2 || q == 3) ? 1 : 0;
							const int xb = (q == 1) ? 2 : (q == 2 || q == 4) ? 1 : 0;
							mma_bf16(tmem + acc1 * (uint32_t)t, smem_desc_sw64(st + (uint32_t)(xa * pa + 32 * sl + 8192 * t)),
							         smem_desc_sw64(st + (uint32_t)(3 * pa + xb * pb + 32 * sl)), id, (k > 0 || sl > 0 || q > 0) ? 1u : 0u);
						}
					}
				mma_commit(&s_empty[s]);
			}
			mma_commit(&s_acc);  // tracks every product issued, also after a failed wait
		}
		__syncwarp();
		if (lane == 0 && !mbar_wait(&s_acc, 0)) *vfail = 1;
		__syncwarp();
	}
	__syncthreads();
	tc_fence_after();
	if (!*vfail && warp < 8) {
		// row of a tile = tensor-memory lane; a warp takes one 32-lane quarter and every other 16 columns
		const int quarter = warp & 3, half = warp >> 2;
		for (int t = 0; t < ntiles; t++) {
			const int row = r0 + 128 * t + 32 * quarter + lane;
			const uint32_t trow = tmem + acc1 * (uint32_t)t + ((uint32_t)(32 * quarter) << 16);
			for (int c0 = 16 * half; c0 < N; c0 += 32) {
				float v[16];
				tmem_ld16(trow + (uint32_t)c0, v);
				if (row >= n) continue;
				float4 *dst = reinterpret_cast<float4 *>(a.A32 + w.aofs + (int64_t)row * np + n0 + c0);
#pragma unroll
				for (int q = 0; q < 4; q++) dst[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
			}
		}
	} else if (*vfail && tid == 0) {
		atomicOr(a.err, 1);
	}
	tc_fence_before();
	__syncthreads();
	if (warp == 0) tmem_dealloc(tmem, ncols);
}

}  // namespace hab200
