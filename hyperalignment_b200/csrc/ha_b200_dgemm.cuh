// ha_b200_dgemm.cuh -- float64 matrix products on the tensor cores (mma.sync m16n8k8 f64, the only
// tensor route for float64) and the blocked ridge solve built on them.
//
// Measured on a B200 with all 148 SMs busy and operands in registers: m16n8k8 f64 37.0 TFLOP/s,
// m8n8k4 36.9, DFMA 28.9; a warp-level product needs 16 shared-memory loads per 8 mma, so shared
// memory stays far from its limit (a 4 x 4 DFMA register tile needs 8 loads per 16 DFMA and is
// bound by it).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "ha_b200_kernels.cuh"

namespace hab200 {

// One CTA of 128 threads computes one 64 x 64 tile; K is staged 16 at a time through kDgStages
// shared-memory stages filled by 8-byte cp.async (rows of gathered time series start at any
// 8-byte address, so wider copies are not always aligned).  Three stages keep two slices in
// flight behind the one being multiplied.
constexpr int kDgThreads = 128;
constexpr int kDgTile = 64;
constexpr int kDgK = 16;
constexpr int kDgStages = 3;
// Operand tile in shared memory: [row][20] when K is contiguous in memory, [k][68] when the row
// index is.  Both strides are 4 (mod 16) doubles, so the fragment reads (8 rows x 4 k per warp) are
// free of bank conflicts.
constexpr int kDgLdK = 20;
constexpr int kDgLdM = 68;
constexpr int kDgOperand = 64 * kDgLdK;  // doubles per operand and stage (the larger of the two layouts)
constexpr size_t kDgSmem = (size_t)kDgStages * 2 * kDgOperand * sizeof(double);

// An operand of the tile product: element (i, k) is at base[(idx ? idx[i] : i) * ld + k] when KC
// (K contiguous), at base[k * ld + i] otherwise.  Rows i >= rows and k >= K read as zero.
struct DgOperand {
	const double *base;
	const int32_t *idx;
	int64_t ld;
	int rows;
};

__device__ __forceinline__ void dg_cp8(double *dst, const double *src, bool ok) {
	const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
	asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(ok ? 8u : 0u) : "memory");
}

// The thread's share of an operand tile: 8 elements of every K slice.
template <bool KC_>
struct DgLoader {
	static constexpr bool KC = KC_;
	const double *p[KC ? 8 : 1];
	int64_t ld;
	uint32_t ok;  // rows inside the operand (KC: one bit per element)
	int k, m;
	__device__ __forceinline__ void init(const DgOperand &o, int i0, int tid) {
		ld = o.ld;
		ok = 0;
		if (KC) {
			k = tid & 15;
			m = tid >> 4;
#pragma unroll
			for (int j = 0; j < 8; j++) {
				const int i = i0 + m + 8 * j;
				const bool in = i < o.rows;
				p[j] = o.base + (in ? (int64_t)(o.idx ? o.idx[i] : i) * o.ld + k : 0);
				ok |= (in ? 1u : 0u) << j;
			}
		} else {
			m = tid & 63;
			k = tid >> 6;
			const bool in = i0 + m < o.rows;
			p[0] = o.base + (in ? i0 + m : 0);
			ok = in ? 1u : 0u;
		}
	}
	__device__ __forceinline__ void load(double *s, int k0, int K, const double *safe) const {
#pragma unroll
		for (int j = 0; j < 8; j++) {
			if (KC) {
				const bool in = ((ok >> j) & 1u) && k0 + k < K;
				dg_cp8(s + (m + 8 * j) * kDgLdK + k, in ? p[j] + k0 : safe, in);
			} else {
				const int kk = k + 2 * j;
				const bool in = ok && k0 + kk < K;
				dg_cp8(s + kk * kDgLdM + m, in ? p[0] + (int64_t)(k0 + kk) * ld : safe, in);
			}
		}
	}
};

template <bool KC>
__device__ __forceinline__ double dg_frag(const double *s, int row, int k) {
	return KC ? s[row * kDgLdK + k] : s[k * kDgLdM + row];
}

__device__ __forceinline__ void dg_mma(double (&c)[4], const double (&a)[4], const double (&b)[2]) {
	asm volatile(
	    "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
	    "{%0, %1, %2, %3};"
	    : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
	    : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

// acc(i, j) += sum_k A(m0 + i, k) B(n0 + j, k) over k in [0, K) for this thread's 32 elements of the
// 64 x 64 tile: warp w covers rows 32 (w & 1).. and columns 32 (w >> 1).., acc[u][v][e] is row
// 16 u + g + 8 (e >> 1), column 8 v + 2 t + (e & 1) of that 32 x 32 block (g = lane / 4, t = lane % 4).
// Ends with a barrier, so the stages may be reused at once.  la and lb load the operands' K slices
// (their rows already placed at m0 and n0); `safe` is any readable address, the source of the
// zero-size copies of elements outside an operand.  cv (shared memory, may be null) scales slice k
// of the product by cv[k].  A warp whose 32 x 32 block lies outside the product (active false) only helps
// to load it.
template <typename LA, typename LB>
__device__ __forceinline__ void dgemm_core(const LA &la, const LB &lb, int K, const double *safe, double *sm,
                                           double (&acc)[2][4][4], bool active = true, const double *cv = nullptr) {
	constexpr bool AKC = LA::KC, BKC = LB::KC;
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	const int g = lane >> 2, t = lane & 3, wm = 32 * (warp & 1), wn = 32 * (warp >> 1);
	const int nk = (K + kDgK - 1) / kDgK;
	auto fill = [&](int s) {
		if (s < nk) {
			double *st = sm + (s % kDgStages) * 2 * kDgOperand;
			la.load(st, s * kDgK, K, safe);
			lb.load(st + kDgOperand, s * kDgK, K, safe);
		}
		asm volatile("cp.async.commit_group;" ::: "memory");
	};
#pragma unroll
	for (int s = 0; s < kDgStages - 1; s++) fill(s);
	for (int s = 0; s < nk; s++) {
		asm volatile("cp.async.wait_group %0;" ::"n"(kDgStages - 2) : "memory");
		__syncthreads();
		fill(s + kDgStages - 1);
		if (!active) continue;
		const double *as = sm + (s % kDgStages) * 2 * kDgOperand, *bs = as + kDgOperand;
#pragma unroll
		for (int kk = 0; kk < kDgK; kk += 8) {
			double a[2][4], b[4][2];
			double c0 = 1.0, c1 = 1.0;
			if (cv) {
				const int k = s * kDgK + kk + t;
				c0 = k < K ? cv[k] : 0.0;
				c1 = k + 4 < K ? cv[k + 4] : 0.0;
			}
#pragma unroll
			for (int u = 0; u < 2; u++)
#pragma unroll
				for (int e = 0; e < 4; e++) {
					a[u][e] = dg_frag<AKC>(as, wm + 16 * u + g + 8 * (e & 1), kk + t + 4 * (e >> 1));
					if (cv) a[u][e] *= e >> 1 ? c1 : c0;
				}
#pragma unroll
			for (int v = 0; v < 4; v++)
#pragma unroll
				for (int e = 0; e < 2; e++) b[v][e] = dg_frag<BKC>(bs, wn + 8 * v + g, kk + t + 4 * e);
#pragma unroll
			for (int u = 0; u < 2; u++)
#pragma unroll
				for (int v = 0; v < 4; v++) dg_mma(acc[u][v], a[u], b[v]);
		}
	}
	asm volatile("cp.async.wait_group 0;" ::: "memory");
	__syncthreads();
}

// Whether the warp's 32 x 32 block of the tile at (m0, n0) holds any element of a rows x cols product.
__device__ __forceinline__ bool dg_active(int m0, int rows, int n0, int cols) {
	const int warp = threadIdx.x >> 5;
	return m0 + 32 * (warp & 1) < rows && n0 + 32 * (warp >> 1) < cols;
}

template <bool AKC, bool BKC>
__device__ __forceinline__ void dgemm_tile(const DgOperand &A, int m0, const DgOperand &B, int n0, int K, double *sm,
                                           double (&acc)[2][4][4]) {
	DgLoader<AKC> la;
	DgLoader<BKC> lb;
	la.init(A, m0, threadIdx.x);
	lb.init(B, n0, threadIdx.x);
	dgemm_core(la, lb, K, A.base, sm, acc, dg_active(m0, A.rows, n0, B.rows));
}

// Lower tile b of a T x T grid: row ti holds ti + 1 tiles.
__device__ __forceinline__ void dg_lower(int b, int &ti, int &tj) {
	ti = 0;
	while (b > ti) b -= ++ti;
	tj = b;
}

__device__ __forceinline__ void dg_zero(double (&acc)[2][4][4]) {
#pragma unroll
	for (int u = 0; u < 2; u++)
#pragma unroll
		for (int v = 0; v < 4; v++)
#pragma unroll
			for (int e = 0; e < 4; e++) acc[u][v][e] = 0.0;
}

// f(i, j, value) for this thread's elements of the tile (i, j in 0..63)
template <typename F>
__device__ __forceinline__ void dg_each(double (&acc)[2][4][4], F f) {
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	const int g = lane >> 2, t = lane & 3, wm = 32 * (warp & 1), wn = 32 * (warp >> 1);
#pragma unroll
	for (int u = 0; u < 2; u++)
#pragma unroll
		for (int v = 0; v < 4; v++)
#pragma unroll
			for (int e = 0; e < 4; e++) f(wm + 16 * u + g + 8 * (e >> 1), wn + 8 * v + 2 * t + (e & 1), acc[u][v][e]);
}

// ---------------------------------------------------------------------------------------------
// ridge  beta_s = (X_s^T X_s + alpha I)^-1 X_s^T Y_s   (csrc/ha_ridge.c:13-54, float64)
// ---------------------------------------------------------------------------------------------
// The reference computes V diag(s / (alpha + s^2)) U^T Y from the thin SVD X_s = U diag(s) V^T; for
// alpha > 0 that is exactly the solution of the regularised normal equations.

// G = X_sl^T X_sl (lower 64 x 64 tiles only, column-major, leading dimension n, at Gscr + aofs) and
// R = X_sl^T Y_sl (all tiles, column j holding right-hand side j, at Rscr + aofs).  One CTA per
// tile: blockIdx.x < T (T + 1) / 2 are the tiles of G, the next T^2 those of R, T = ceil(n / 64);
// the grid is sized for the widest searchlight of the launch.
__global__ void __launch_bounds__(kDgThreads) k_ridge_gram(const SlWork *__restrict__ work, const int32_t *__restrict__ sl_idx,
                                                           const double *__restrict__ X, const double *__restrict__ Y, int nt,
                                                           double *__restrict__ Gscr, double *__restrict__ Rscr) {
	extern __shared__ __align__(16) double dg_sm[];
	const SlWork w = work[blockIdx.y];
	const int n = w.n, T = (n + kDgTile - 1) / kDgTile, low = T * (T + 1) / 2;
	int b = blockIdx.x;
	if (b >= low + T * T) return;
	const bool gram = b < low;
	int ti, tj;
	if (gram) {
		dg_lower(b, ti, tj);
	} else {
		b -= low;
		ti = b % T;
		tj = b / T;
	}
	const int32_t *sl = sl_idx + w.sofs;
	double acc[2][4][4];
	dg_zero(acc);
	const DgOperand A = {X, sl, nt, n}, B = {gram ? X : Y, sl, nt, n};
	const int i0 = ti * kDgTile, j0 = tj * kDgTile;
	dgemm_tile<true, true>(A, i0, B, j0, nt, dg_sm, acc);
	double *out = (gram ? Gscr : Rscr) + w.aofs;
	dg_each(acc, [&](int i, int j, double v) {
		if (i0 + i < n && j0 + j < n) out[(int64_t)(j0 + j) * n + i0 + i] = v;
	});
}

// The solve, one CTA per searchlight: left-looking Cholesky of G + alpha I in panels of 64 columns
// with the right-hand sides as extra rows, so the forward solve is the same tile product; each
// diagonal block's inverse W_k replaces the triangular solves by products with it (and is kept
// in the diagonal block of G for the backward solve).  All O(n^3) work runs on the float64 tensor
// cores; what is serial is the 64 x 64 factor and inverse of each panel, which overlaps the
// products of the SM's other CTA.  2,562 searchlights of 100-300 vertices (nt = 400) take 14.5 ms
// with the reduction; a column-at-a-time factor and solve, one dependent pass over the trailing
// block per column, took 168 ms.  beta is written (float64) in the T
// layout: row-major for CSR output (row i = source vertex i), column-major for CSC output.  A
// non-positive pivot (alpha = 0 with a rank-deficient X_s) marks the searchlight kFlagUnconverged and
// writes zeros.
constexpr size_t kRidgeSmem = kDgSmem + (size_t)kDgTile * kDgLdM * sizeof(double);

// T <- T Q for a 64 x 64 tile in shared memory (row-major, leading dimension 68), Q(k, j) = W[j][k]
// (TRANS) or W[k][j]; the product is left in acc.
template <bool TRANS>
__device__ __forceinline__ void dg_tile_mul(const double *Ts, const double *W, double (&acc)[2][4][4]) {
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	const int g = lane >> 2, t = lane & 3, wm = 32 * (warp & 1), wn = 32 * (warp >> 1);
	dg_zero(acc);
#pragma unroll 2
	for (int kk = 0; kk < kDgTile; kk += 8) {
		double a[2][4], b[4][2];
#pragma unroll
		for (int u = 0; u < 2; u++)
#pragma unroll
			for (int e = 0; e < 4; e++) a[u][e] = Ts[(wm + 16 * u + g + 8 * (e & 1)) * kDgLdM + kk + t + 4 * (e >> 1)];
#pragma unroll
		for (int v = 0; v < 4; v++)
#pragma unroll
			for (int e = 0; e < 2; e++) {
				const int j = wn + 8 * v + g, k = kk + t + 4 * e;
				b[v][e] = TRANS ? W[j * kDgLdM + k] : W[k * kDgLdM + j];
			}
#pragma unroll
		for (int u = 0; u < 2; u++)
#pragma unroll
			for (int v = 0; v < 4; v++) dg_mma(acc[u][v], a[u], b[v]);
	}
}

// W = L^-1 (row-major, leading dimension 68, zero above the diagonal) of the Cholesky factor L of a
// symmetric 64 x 64 block S (both triangles).  Two threads a row, the row in registers: at step k
// row k goes to W unscaled, and every later row r takes f = S(r, k) / d_k times it off, with its own
// entry k replaced by -f; that leaves the Schur complement right of k and the rows of L^-1 (times
// sqrt(d)) left of it.  One barrier and 32 multiply-adds a thread per step.  The registers are rotated
// by one column quad every four steps, so the entry being replaced has a fixed register.  Returns
// whether this thread saw a pivot that is not positive.
__device__ __forceinline__ bool dg_chol_inverse(const double *S, double *W) {
	const int r = threadIdx.x >> 1, h = threadIdx.x & 1;
	double m[32];  // m[2 i + e] = S(r, 4 ((quad + i) % 16) + 2 h + e)
#pragma unroll
	for (int i = 0; i < 16; i++) {
		m[2 * i] = S[r * kDgLdM + 4 * i + 2 * h];
		m[2 * i + 1] = S[r * kDgLdM + 4 * i + 2 * h + 1];
	}
	bool bad = false;
	for (int quad = 0; quad < 16; quad++) {
#pragma unroll
		for (int kk = 0; kk < 4; kk++) {
			const int k = 4 * quad + kk;
			double *wk = W + k * kDgLdM;
			if (r == k) {
#pragma unroll
				for (int i = 0; i < 16; i++)
					*reinterpret_cast<double2 *>(wk + 4 * ((quad + i) & 15) + 2 * h) = make_double2(m[2 * i], m[2 * i + 1]);
			}
			__syncthreads();
			const double d = wk[k];
			bad = bad || !(d > 0.0);
			if (r > k) {
				const double f = wk[r] / d;
#pragma unroll
				for (int i = 0; i < 16; i++) {
					const double2 x = *reinterpret_cast<const double2 *>(wk + 4 * ((quad + i) & 15) + 2 * h);
					m[2 * i] -= f * x.x;
					m[2 * i + 1] -= f * x.y;
				}
				if (h == kk >> 1) m[kk & 1] = -f;
			}
		}
		const double m0 = m[0], m1 = m[1];
#pragma unroll
		for (int i = 0; i < 30; i++) m[i] = m[i + 2];
		m[30] = m0;
		m[31] = m1;
	}
	__syncthreads();
	const double p = rsqrt(W[r * kDgLdM + r]);
	__syncthreads();
	for (int c = h; c < kDgTile; c += 2) {
		double &x = W[r * kDgLdM + c];
		x = c < r ? x * p : (c == r ? p : 0.0);
	}
	return bad;
}

__global__ void __launch_bounds__(kDgThreads) k_ridge_chol(const SlWork *__restrict__ work, double *__restrict__ Gscr,
                                                           double *__restrict__ Rscr, double *__restrict__ Bout,
                                                           double alpha, int t_rowmajor, SlStats *__restrict__ stats) {
	extern __shared__ __align__(16) double dg_sm[];
	double *Ts = dg_sm;  // aliases the stages, which are idle while it is used
	double *W = dg_sm + kDgSmem / sizeof(double);
	__shared__ int bad;
	const SlWork w = work[blockIdx.x];
	const int n = w.n, T = (n + kDgTile - 1) / kDgTile, tid = threadIdx.x;
	double *G = Gscr + w.aofs;  // G[c * n + r] = G(r, c); lower triangle used
	double *R = Rscr + w.aofs;  // R[j * n + i] = rhs(i, j)
	double acc[2][4][4];
	if (tid == 0) bad = 0;
	for (int kb = 0; kb < T; kb++) {
		const int k0 = kb * kDgTile, nb = min(kDgTile, n - k0);
		const DgOperand Lk = {G + k0, nullptr, n, n - k0};  // rows k0.. of the factor, columns [0, k0)
		// diagonal block
		dg_zero(acc);
		dgemm_tile<false, false>(Lk, 0, Lk, 0, k0, dg_sm, acc);
		dg_each(acc, [&](int i, int j, double v) {
			double x = i == j ? 1.0 : 0.0;  // identity padding
			if (i < nb && j < nb) x = G[(int64_t)(k0 + min(i, j)) * n + k0 + max(i, j)] - v + (i == j ? alpha : 0.0);
			Ts[i * kDgLdM + j] = x;
		});
		__syncthreads();
		if (dg_chol_inverse(Ts, W)) bad = 1;
		__syncthreads();
		for (int e = tid; e < nb * nb; e += kDgThreads) {
			const int j = e / nb, i = e - j * nb;
			G[(int64_t)(k0 + j) * n + k0 + i] = W[i * kDgLdM + j];
		}
		__syncthreads();
		// rows below, then the right-hand sides as rows: L(i, k) = (A(i, k) - sum) W^T
		for (int it = kb + 1; it < T + T; it++) {
			const bool rhs = it >= T;
			const int i0 = rhs ? (it - T) * kDgTile : it * kDgTile;
			dg_zero(acc);
			if (rhs)
				dgemm_tile<true, false>(DgOperand{R, nullptr, n, n}, i0, Lk, 0, k0, dg_sm, acc);
			else
				dgemm_tile<false, false>(DgOperand{G, nullptr, n, n}, i0, Lk, 0, k0, dg_sm, acc);
			dg_each(acc, [&](int i, int j, double v) {
				double x = 0.0;
				if (i0 + i < n && j < nb)
					x = (rhs ? R[(int64_t)(i0 + i) * n + k0 + j] : G[(int64_t)(k0 + j) * n + i0 + i]) - v;
				Ts[i * kDgLdM + j] = x;
			});
			__syncthreads();
			dg_tile_mul<true>(Ts, W, acc);
			dg_each(acc, [&](int i, int j, double v) {
				if (i0 + i >= n || j >= nb) return;
				if (rhs) R[(int64_t)(i0 + i) * n + k0 + j] = v;
				else G[(int64_t)(k0 + j) * n + i0 + i] = v;
			});
			__syncthreads();
		}
	}
	// backward solve, right-hand sides as rows: beta(j, k) = (Z(j, k) - sum_{i > k} beta(j, i) L(i, k)) W_k
	double *Bo = Bout + w.tofs;
	const int64_t ti = t_rowmajor ? n : 1, tj = t_rowmajor ? 1 : n;
	for (int kb = T - 1; kb >= 0; kb--) {
		const int k0 = kb * kDgTile, nb = min(kDgTile, n - k0), k1 = k0 + nb;
		for (int e = tid; e < kDgTile * kDgTile; e += kDgThreads) {
			const int j = e >> 6, i = e & 63;
			W[i * kDgLdM + j] = (i < nb && j < nb) ? G[(int64_t)(k0 + j) * n + k0 + i] : 0.0;
		}
		for (int jt = 0; jt < T; jt++) {
			const int i0 = jt * kDgTile;
			dg_zero(acc);
			dgemm_tile<true, true>(DgOperand{R + k1, nullptr, n, n}, i0, DgOperand{G + (int64_t)k0 * n + k1, nullptr, n, nb},
			                       0, n - k1, dg_sm, acc);
			dg_each(acc, [&](int i, int j, double v) {
				Ts[i * kDgLdM + j] = (i0 + i < n && j < nb) ? R[(int64_t)(i0 + i) * n + k0 + j] - v : 0.0;
			});
			__syncthreads();
			dg_tile_mul<false>(Ts, W, acc);
			const bool zero = bad != 0;
			dg_each(acc, [&](int i, int j, double v) {
				if (i0 + i >= n || j >= nb) return;
				R[(int64_t)(i0 + i) * n + k0 + j] = v;
				Bo[(int64_t)(k0 + j) * ti + (int64_t)(i0 + i) * tj] = zero ? 0.0 : v;
			});
			__syncthreads();
		}
	}
	if (tid == 0) {
		SlStats st = stats[w.slot];
		st.s_sum = 0.0;
		st.flags = bad ? (kFlagUnconverged | kFlagFP64) : kFlagFP64;
		stats[w.slot] = st;
	}
}

}  // namespace hab200
