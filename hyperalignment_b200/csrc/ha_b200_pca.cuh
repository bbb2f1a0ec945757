// ha_b200_pca.cuh -- searchlight PCA template (src/hyperalignment/searchlight.py:215-236 with
// compute_template(kind="pca", max_npc=n, common_topography=True, demean=False),
// src/hyperalignment/local_template.py:224-248, :72-78, :11-53), float64 throughout.
//
// Per searchlight s with vertices sl (n of them, n <= nt) and ns subjects D_j (nt x nv):
//   X = [D_1[:, sl], ..., D_ns[:, sl]]                     nt x ns n
//   the top n singular pairs of X from the smaller Gram (m = min(nt, ns n) <= 512):
//     time side   (m = nt):   X X^T = U diag(lambda) U^T,   tmpl = U_n diag(sqrt(lambda_n)) / sqrt(ns)
//     vertex side (m = ns n): X^T X = W diag(lambda) W^T,   tmpl = X W_n / sqrt(ns)
//   both by pivoted Cholesky and one-sided Jacobi (k_pchol, k_jacobi); then M = sum_j D_j[:, sl],
//   R = polar(tmpl^T M) by the float64 Newton-Schulz iteration (ha_b200_polar.cuh), and
//   template[:, sl] += (tmpl R) diag(w_s) with the searchlight weights, reduced per vertex in
//   searchlight order.
// tmpl R depends only on the top-n singular subspace of X (signs and rotations inside a degenerate
// eigenspace cancel in tmpl polar(tmpl^T M)), so this exact route agrees with the reference's
// randomized SVD wherever that subspace is separated from the rest.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "ha_b200_dgemm.cuh"

namespace hab200 {

constexpr int kPcaMaxM = 512;  // Gram order limit (the pivoted Cholesky's rank arrays and the widest Jacobi instance)

// Per-searchlight scratch of the PCA template (float64 elements from the searchlight's base):
// tmpl (nt x n), M (nt x n), then a work area that first holds the gathered X (nt x m) and the
// selected eigenvectors (m x n, vertex side) and finally C = tmpl R (nt x n).  All column-major.
struct PcaLayout {
	int64_t tmpl, M, work, wsel, total;
	__host__ __device__ static PcaLayout make(int nt, int n, int m, bool vertex_side) {
		PcaLayout L;
		const int64_t tn = (int64_t)nt * n;
		L.tmpl = 0;
		L.M = tn;
		L.work = 2 * tn;
		L.wsel = L.work + (int64_t)nt * m;
		const int64_t w = vertex_side ? (int64_t)nt * m + (int64_t)m * n : tn;
		L.total = (L.work + (w > tn ? w : tn) + 31) & ~(int64_t)31;
		return L;
	}
};

// Column offsets of X: column k = j n + a is subject j's vertex sl[a].
__device__ __forceinline__ int64_t pca_col(const int32_t *sl, int n, int64_t plane, int nt, int k) {
	const int j = k / n;
	return (int64_t)j * plane + (int64_t)sl[k - j * n] * nt;
}

// Loader of X for the tile products (DgLoader's slices): row i of the operand is time point i (time
// side: K runs over the columns of X, rows contiguous) or column i of X (vertex side: K runs over
// time, K contiguous).
template <bool TSIDE>
struct PcaLoader {
	static constexpr bool KC = !TSIDE;
	const double *D;
	const int32_t *sl;
	int64_t plane;
	int n, nt, rows, i0, m, k;
	const double *p[TSIDE ? 1 : 8];
	uint32_t ok;
	__device__ __forceinline__ void init(const double *D_, const int32_t *sl_, int n_, int64_t plane_, int nt_, int rows_,
	                                     int i0_) {
		D = D_; sl = sl_; n = n_; plane = plane_; nt = nt_; rows = rows_; i0 = i0_;
		ok = 0;
		if (TSIDE) {
			m = threadIdx.x & 63;
			k = threadIdx.x >> 6;
			ok = i0 + m < rows ? 1u : 0u;
			p[0] = D + i0 + m;
		} else {
			k = threadIdx.x & 15;
			m = threadIdx.x >> 4;
#pragma unroll
			for (int j = 0; j < 8; j++) {
				const int i = i0 + m + 8 * j;
				const bool in = i < rows;
				p[j] = D + (in ? pca_col(sl, n, plane, nt, i) : 0) + k;
				ok |= (in ? 1u : 0u) << j;
			}
		}
	}
	__device__ __forceinline__ void load(double *s, int k0, int K, const double *safe) const {
#pragma unroll
		for (int j = 0; j < 8; j++) {
			if (TSIDE) {
				const int kk = k + 2 * j;
				const bool in = ok && k0 + kk < K;
				dg_cp8(s + kk * kDgLdM + m, in ? p[0] + pca_col(sl, n, plane, nt, k0 + kk) : safe, in);
			} else {
				const bool in = ((ok >> j) & 1u) && k0 + k < K;
				dg_cp8(s + (m + 8 * j) * kDgLdK + k, in ? p[j] + k0 : safe, in);
			}
		}
	}
};

// The Gram of every searchlight of a batch into the V scratch at wm.aofs (lower 64 x 64 tiles of
// m x m, leading dimension m, wm.n = m): X X^T (m = nt, reduction over the ns n columns) or X^T X
// (m = ns n < nt, reduction over time), one CTA per tile.
__global__ void __launch_bounds__(kDgThreads) k_pca_gram(const SlWork *__restrict__ wm, const int32_t *__restrict__ sl_idx,
                                                         const int32_t *__restrict__ off, const double *__restrict__ D,
                                                         int ns, int nt, int nv, double *__restrict__ Gscr) {
	extern __shared__ __align__(16) double dg_sm[];
	const SlWork w = wm[blockIdx.y];
	const int n = off[w.s + 1] - off[w.s], m = w.n;
	const int T = (m + kDgTile - 1) / kDgTile;
	if ((int)blockIdx.x >= T * (T + 1) / 2) return;
	int ti, tj;
	dg_lower(blockIdx.x, ti, tj);
	const int i0 = ti * kDgTile, j0 = tj * kDgTile;
	const int32_t *sl = sl_idx + off[w.s];
	const int64_t plane = (int64_t)nt * nv;
	double acc[2][4][4];
	dg_zero(acc);
	if (m == nt) {
		PcaLoader<true> la, lb;
		la.init(D, sl, n, plane, nt, m, i0);
		lb.init(D, sl, n, plane, nt, m, j0);
		dgemm_core(la, lb, ns * n, D, dg_sm, acc, dg_active(i0, m, j0, m));
	} else {
		PcaLoader<false> la, lb;
		la.init(D, sl, n, plane, nt, m, i0);
		lb.init(D, sl, n, plane, nt, m, j0);
		dgemm_core(la, lb, nt, D, dg_sm, acc, dg_active(i0, m, j0, m));
	}
	double *G = Gscr + w.aofs;
	dg_each(acc, [&](int i, int j, double v) {
		if (i0 + i >= m || j0 + j >= m) return;
		G[(int64_t)(j0 + j) * m + i0 + i] = v;
		if (i0 != j0) G[(int64_t)(i0 + i) * m + j0 + j] = v;
	});
}

// The template of every searchlight of a batch and the subjects' sum M.  Eigenvectors (V scratch at wm.aofs, column-major, leading dimension m) and
// eigenvalues (uv + wm.uvofs) from the eigen decomposition; the n largest eigenvalues (ties:
// the lower column) are taken in decreasing order.  wm and wn (the polar work items) are in slot
// order.
__global__ void __launch_bounds__(256) k_pca_tmpl(const SlWork *__restrict__ wm, const SlWork *__restrict__ wn,
                                                  const int32_t *__restrict__ sl_idx, const double *__restrict__ D,
                                                  int ns, int nt, int nv, const double *__restrict__ Vscr,
                                                  const double *__restrict__ uv, const int64_t *__restrict__ pofs,
                                                  double *__restrict__ Pscr) {
	const SlWork em = wm[blockIdx.x];
	const SlWork ep = wn[blockIdx.x];
	const int n = ep.n, m = em.n;
	const bool tside = (m == nt);
	const int32_t *sl = sl_idx + ep.sofs;
	const double *U = Vscr + em.aofs;
	const double *lam = uv + em.uvofs;
	const PcaLayout L = PcaLayout::make(nt, n, m, !tside);
	double *base = Pscr + pofs[ep.slot];
	double *tmpl = base + L.tmpl;
	double *M = base + L.M;
	__shared__ int sel[kPcaMaxM];
	__shared__ double ps[16][65], qs[16][65];
	for (int c = threadIdx.x; c < m; c += blockDim.x) {
		const double lc = lam[c];
		int rank = 0;
		for (int c2 = 0; c2 < m; c2++) {
			const double l2 = lam[c2];
			rank += (l2 > lc || (l2 == lc && c2 < c)) ? 1 : 0;
		}
		if (rank < n) sel[rank] = c;
	}
	__syncthreads();
	const double inv_ns = rsqrt((double)ns);
	const int64_t plane = (int64_t)nt * nv;
	for (int64_t e = threadIdx.x; e < (int64_t)nt * n; e += blockDim.x) {
		const int r = (int)(e / nt), t = (int)(e - (int64_t)r * nt);
		if (tside) {
			const int c = sel[r];
			tmpl[e] = U[(int64_t)c * m + t] * sqrt(fmax(lam[c], 0.0)) * inv_ns;
		}
		double s = 0.0;
		for (int j = 0; j < ns; j++) s += D[(int64_t)j * plane + (int64_t)sl[r] * nt + t];
		M[e] = s;
	}
	if (!tside) {
		// tmpl = X W_sel / sqrt(ns): X gathered (nt x m) and the selected eigenvectors (m x n)
		double *Xg = base + L.work;
		double *Ws = base + L.wsel;
		for (int64_t e = threadIdx.x; e < (int64_t)nt * m; e += blockDim.x) {
			const int k = (int)(e / nt), t = (int)(e - (int64_t)k * nt);
			Xg[e] = D[pca_col(sl, n, plane, nt, k) + t];
		}
		for (int64_t e = threadIdx.x; e < (int64_t)m * n; e += blockDim.x) {
			const int r = (int)(e / m), k = (int)(e - (int64_t)r * m);
			Ws[e] = U[(int64_t)sel[r] * m + k];
		}
		__syncthreads();
		// tmpl(t, r) = sum_k Xg(t, k) Ws(k, r) / sqrt(ns)
		GemmArgs<double, double> g;
		g.M = nt; g.N = n; g.K = m;
		g.P = Xg; g.pk = nt; g.pi = 1;
		g.Q = Ws; g.qk = 1; g.qj = m;
		g.d = nullptr; g.alpha = inv_ns;
		g.E = nullptr; g.ei = 0; g.ej = 0; g.beta = 0.0;
		g.C = tmpl; g.ci = 1; g.cj = nt;
		block_gemm(g, ps, qs);
	}
}

// B = tmpl^T M (n x n), the matrix whose polar factor rotates the template, into the polar solve's A
// region at wn.aofs with the padding columns of its block layout zero.  One CTA per 64 x 64 tile.
__global__ void __launch_bounds__(kDgThreads) k_pca_b(const SlWork *__restrict__ wm, const SlWork *__restrict__ wn, int nt,
                                                      const int64_t *__restrict__ pofs, const double *__restrict__ Pscr,
                                                      double *__restrict__ Ascr) {
	extern __shared__ __align__(16) double dg_sm[];
	const SlWork ep = wn[blockIdx.y];
	const int n = ep.n, m = wm[blockIdx.y].n, T = (n + kDgTile - 1) / kDgTile;
	if ((int)blockIdx.x >= T * T) return;
	const PcaLayout L = PcaLayout::make(nt, n, m, m != nt);
	const double *base = Pscr + pofs[ep.slot];
	const int i0 = ((int)blockIdx.x % T) * kDgTile, j0 = ((int)blockIdx.x / T) * kDgTile;
	double acc[2][4][4];
	dg_zero(acc);
	dgemm_tile<true, true>(DgOperand{base + L.tmpl, nullptr, nt, n}, i0, DgOperand{base + L.M, nullptr, nt, n}, j0, nt, dg_sm, acc);
	double *A = Ascr + ep.aofs;
	dg_each(acc, [&](int i, int j, double v) {
		if (i0 + i < n && j0 + j < n) A[(int64_t)(j0 + j) * n + i0 + i] = v;
	});
	if (blockIdx.x == 0)
		for (int64_t e = (int64_t)n * n + threadIdx.x; e < (int64_t)n * ep.nblk * ep.bsz; e += blockDim.x) A[e] = 0.0;
}

// The polar factors R (float, column-major in the T scratch at wn.tofs) as float64 in the M block
// (M is no longer needed).
__global__ void __launch_bounds__(256) k_pca_widen(const SlWork *__restrict__ wm, const SlWork *__restrict__ wn,
                                                   const float *__restrict__ Tscr, int nt,
                                                   const int64_t *__restrict__ pofs, double *__restrict__ Pscr) {
	const SlWork ep = wn[blockIdx.x];
	const int n = ep.n, m = wm[blockIdx.x].n;
	double *Rd = Pscr + pofs[ep.slot] + PcaLayout::make(nt, n, m, m != nt).M;
	const float *R = Tscr + ep.tofs;
	for (int64_t e = threadIdx.x; e < (int64_t)n * n; e += blockDim.x) Rd[e] = (double)R[e];
}

// C = tmpl R (nt x n, into the work area), one CTA per 64 x 64 tile.  wn in slot order; m of the slot's
// Gram from wm (slot order).
__global__ void __launch_bounds__(kDgThreads) k_pca_contrib(const SlWork *__restrict__ wm, const SlWork *__restrict__ wn,
                                                            int nt, const int64_t *__restrict__ pofs,
                                                            double *__restrict__ Pscr) {
	extern __shared__ __align__(16) double dg_sm[];
	const SlWork ep = wn[blockIdx.y];
	const int n = ep.n, m = wm[blockIdx.y].n;
	const int Tt = (nt + kDgTile - 1) / kDgTile, T = (n + kDgTile - 1) / kDgTile;
	if ((int)blockIdx.x >= Tt * T) return;
	const PcaLayout L = PcaLayout::make(nt, n, m, m != nt);
	double *base = Pscr + pofs[ep.slot];
	const int i0 = ((int)blockIdx.x % Tt) * kDgTile, j0 = ((int)blockIdx.x / Tt) * kDgTile;
	double acc[2][4][4];
	dg_zero(acc);
	// C(t, j) = sum_i tmpl(t, i) R(i, j)
	dgemm_tile<false, true>(DgOperand{base + L.tmpl, nullptr, nt, nt}, i0, DgOperand{base + L.M, nullptr, n, n}, j0, n, dg_sm, acc);
	double *C = base + L.work;
	dg_each(acc, [&](int i, int j, double v) {
		if (i0 + i < nt && j0 + j < n) C[(int64_t)(j0 + j) * nt + i0 + i] = v;
	});
}

// template[:, v] += sum over the searchlights s of [s_lo, s_hi) holding v (member a), in
// searchlight order, of w_s[a] C_s[:, a] (w = 1 without weights).  One CTA per vertex, threads
// over time; pofs and the Gram orders mg are per slot s - s_lo.
__global__ void __launch_bounds__(256) k_pca_reduce(const int64_t *__restrict__ vl_ptr, const int2 *__restrict__ vl_ent,
                                                    const int32_t *__restrict__ off, const double *__restrict__ wts,
                                                    const int64_t *__restrict__ pofs, const int32_t *__restrict__ mg,
                                                    const double *__restrict__ Pscr, int nt, int s_lo, int s_hi,
                                                    double *__restrict__ tpl) {
	const int v = blockIdx.x;
	double *out = tpl + (int64_t)v * nt;
	for (int64_t k = vl_ptr[v]; k < vl_ptr[v + 1]; k++) {
		const int2 e = vl_ent[k];
		if (e.x < s_lo || e.x >= s_hi) continue;
		const int n = off[e.x + 1] - off[e.x];
		const double wv = wts ? wts[off[e.x] + e.y] : 1.0;
		const PcaLayout L = PcaLayout::make(nt, n, mg[e.x - s_lo], mg[e.x - s_lo] != nt);
		const double *C = Pscr + pofs[e.x - s_lo] + L.work + (int64_t)e.y * nt;
		for (int t = threadIdx.x; t < nt; t += blockDim.x) out[t] += wv * C[t];
	}
}

}  // namespace hab200
