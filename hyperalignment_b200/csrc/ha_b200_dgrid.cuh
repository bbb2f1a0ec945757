// ha_b200_dgrid.cuh -- the ridge grid search of ha_b200_grid.cuh in float64 (the same composition of
// csrc/ha_ridge.c:97-345 and the same winners), arranged for the float64 tensor cores.
//
// Everything is a batch over (searchlight, CV model) items:
//   * a model's training rows are a bootstrap, so only its d distinct rows are gathered, scaled by the
//     square root of their multiplicity (5-fold splits of 500 rows keep about 220 of 500): X_d, Y_d;
//   * the eigen decomposition runs on the smaller of two matrices with the same nonzero eigenvalues,
//     p = min(n, d): the Gram matrix G = X_d^T X_d = V L V^T when n <= d, the kernel matrix
//     X_d X_d^T = U L U^T otherwise;
//   * with W = X_d V, Q = W^T Y_d, E = X_te V, N = V in the first form and Q = U^T Y_d,
//     E = X_te X_d^T U, N = X_d^T U in the second, component k contributes E_k q_k^T / (alpha + l_k) to
//     the test predictions and N_k q_k^T / (alpha + l_k) to beta: the second form divides by no
//     singular value;
//   * the eigenvalues are taken again as the squared column norms of W or N, the singular values of
//     X_d itself: those of the Gram matrix carry an error of eps l_max whatever their size, which at
//     alpha = 1e-3 and n = d (singular values down to 1e-5 of the largest) left costs 1e-9 off;
//   * a grid point's cost is accumulated in the registers that hold the predictions (they start at
//     -Y, and every PC chunk adds its components), so predictions go to memory only for the rows that
//     several models test, whose average is formed afterwards.
// Badly scaled searchlights are left to ha_b200_grid.cuh (k_dg_scaled).
// All products are 64 x 64 tiles, one CTA a tile.  512 searchlights of 50-500 vertices, 500 rows, 5 folds,
// 10 penalties x 4 PC counts: 89 ms (eigen solves 41, evaluation 28, other products 17); one CTA a
// searchlight with Jacobi eigen solves on the n x n Gram matrices took 835 ms, and its costs were up to
// 1.7e-10 off where these are within 1.6e-11.
#pragma once

#include "ha_b200_dgemm.cuh"
#include "ha_b200_eig.cuh"
#include "ha_b200_grid.cuh"

namespace hab200 {

// A CV model: its distinct training rows drow / dsq [d_ofs, d_ofs + d_n) and its test rows
// terow / tew [te_ofs, te_ofs + te_n), the te1 rows that no other model tests first.  The others are the
// searchlight's entries entry0, entry0 + 1, .. of predictions to be averaged.
struct DgModel {
	int32_t d_ofs, d_n, te_ofs, te_n, te1, entry0;
};

struct DgParams {
	const DgModel *mdl;
	const int32_t *drow;
	const double *dsq;
	const int32_t *terow;
	const double *tew;      // 1 / (number of models that test the row)
	const int32_t *ovrow;   // rows tested by several models, nov
	const int32_t *ovptr;   // nov + 1: the row's entries in ovent
	const int32_t *ovent;
	const int32_t *untested;
	const double *alphas;
	const int32_t *npcs;
	int models, nt, n_alphas, n_npcs, nov, entries, n_untested;
	int model0;             // host: position of mdl[0] in the plan's list of models
};

// One (searchlight, model): offsets into the grid scratch (float64 elements).
struct DgItem {
	int64_t xd, yd, xte, yte;  // d x n, d x n, te x n, te x n, column-major
	int64_t g;                 // p x p matrix, then its eigenvectors
	int64_t c;                 // n <= d: W = X_d V (d x p); else X_te X_d^T (te x d); column-major
	int64_t q;                 // p x n; before that the eigen solver's p x p basis
	int64_t e;                 // te x p, row-major, scaled by the test weights
	int64_t nv;                // n x p (n <= d: the eigenvectors themselves)
	int64_t lam;               // p
	int32_t n, p, dual, model;
	int32_t sofs, sl;          // flat offset of the searchlight's vertices, its position in the batch
	int32_t part0, pad_;       // first cost partial of the item within the searchlight
};

// One searchlight of the batch.
struct DgSl {
	int64_t yov;    // targets on the several-model rows, [row][n]
	int64_t pov;    // predictions of the entries, [grid point of the current penalties][entry][n]
	int64_t part;   // cost partials, [grid point][nparts]
	int64_t cost;   // [grid point]
	int64_t tofs;   // beta in the float64 T scratch
	int32_t s, n, item0, nparts;
	int32_t sofs, pad_;
};

// Squared norms of X's columns over every model's distinct training rows (with their multiplicities), a warp
// a (vertex, model).
__global__ void __launch_bounds__(256) k_dg_norms(const double *__restrict__ X, int nv, const DgParams dp,
                                                  double *__restrict__ norms) {
	const int v = (int)blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31, m = (int)blockIdx.y;
	if (v >= nv) return;
	const DgModel md = dp.mdl[m];
	const double *x = X + (int64_t)v * dp.nt;
	double s = 0.0;
	for (int t = lane; t < md.d_n; t += 32) {
		const double y = dp.dsq[md.d_ofs + t] * x[dp.drow[md.d_ofs + t]];
		s = fma(y, y, s);
	}
	s = warp_sum(s);
	if (lane == 0) norms[(int64_t)m * nv + v] = s;
}

// Whether the nonzero columns of a searchlight differ in norm by more than kDgMaxScale over the rows of some
// model, or are not finite (or beyond the range below), a warp a searchlight.  The tridiagonal reduction's error is eps ||G||, whatever
// a column's own size, and the kernel matrix keeps no column scale at all, so both lose the square of the
// ratio; pivoted Cholesky and one-sided Jacobi are accurate relative to every column and take such
// searchlights.  Error of beta at alpha = 1e-3, tile products / Jacobi, median over ten draws of 120 x 60,
// 60 x 120 and 100 x 100 with some columns scaled by r: 3.9e-15 / 1.1e-14, 3.6e-15 / 1.2e-14 and 4.1e-12 /
// 2.5e-12 at r = 1; 3.1e-14 / 2.2e-14, 2.7e-14 / 2.0e-14 and 8.1e-12 / 1.2e-12 at 8; 8.1e-13 / 9.0e-14, 3.8e-13 /
// 6.2e-14 and 1.7e-10 / 9.4e-12 at 32; at 1e4 up to 1e-4 / 2e-8.  z-scored series lie below 2 over the rows of
// a bootstrap and series with a standard deviation of 1.02-6.1 over the sphere below 6.1; the way by Jacobi
// takes nine times as long (512 searchlights of 50-500 vertices: 835 against 89 ms).
// So do searchlights whose squared norms leave 1e-100 .. 1e100: the reduction squares entries of G, which from
// 2^256 times unit columns on overflowed (and at 2^-270 vanished); Jacobi gives the same bits there up to 2^500.
constexpr double kDgMaxScale = 8.0, kDgMinNorm = 1e-100, kDgMaxNorm = 1e100;
__global__ void __launch_bounds__(256) k_dg_scaled(const int32_t *__restrict__ off, const int32_t *__restrict__ sl_idx, int count,
                                                   int nv, int models, const double *__restrict__ norms,
                                                   int32_t *__restrict__ scaled) {
	const int s = (int)blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
	if (s >= count) return;
	bool bad = false;
	for (int m = 0; m < models; m++) {
		double mn = INFINITY, mx = 0.0;
		for (int i = off[s] + lane; i < off[s + 1]; i += 32) {
			const double x = norms[(int64_t)m * nv + sl_idx[i]];
			if (x > 0.0) mn = fmin(mn, x);
			mx = fmax(mx, x);
			bad = bad || !(x <= kDgMaxNorm);
		}
		for (int o = 16; o > 0; o >>= 1) {
			mn = fmin(mn, __shfl_xor_sync(0xffffffffu, mn, o));
			mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
		}
		bad = bad || mx > kDgMaxScale * kDgMaxScale * mn || (mx > 0.0 && mx < kDgMinNorm);
	}
	bad = __any_sync(0xffffffffu, bad);
	if (lane == 0) scaled[s] = bad ? 1 : 0;
}

// Gathered rows of one item (Y may be null when there are no test rows): the distinct training rows of X and Y, the test rows of X and Y, and (by
// the first model's CTA) the targets of the several-model rows.
__global__ void __launch_bounds__(256) k_dg_gather(const DgItem *__restrict__ items, const DgSl *__restrict__ sls,
                                                   const int32_t *__restrict__ sl_idx, const double *__restrict__ X,
                                                   const double *__restrict__ Y, double *__restrict__ S, const DgParams dp) {
	const DgItem it = items[blockIdx.x];
	const DgModel md = dp.mdl[it.model];
	const int32_t *sl = sl_idx + it.sofs;
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	for (int v = warp; v < it.n; v += 8) {  // a warp a vertex: the rows ascend, so its reads stay in few lines
		const double *x = X + (int64_t)sl[v] * dp.nt, *y = Y ? Y + (int64_t)sl[v] * dp.nt : nullptr;
		for (int t = lane; t < md.d_n; t += 32) {
			const int r = dp.drow[md.d_ofs + t];
			const double w = dp.dsq[md.d_ofs + t];
			S[it.xd + (int64_t)v * md.d_n + t] = w * x[r];
			if (Y) S[it.yd + (int64_t)v * md.d_n + t] = w * y[r];
		}
		for (int t = lane; t < md.te_n; t += 32) {
			const int r = dp.terow[md.te_ofs + t];
			S[it.xte + (int64_t)v * md.te_n + t] = x[r];
			S[it.yte + (int64_t)v * md.te_n + t] = y[r];
		}
		if (it.model == 0) {
			const int64_t yov = sls[it.sl].yov + v;
			for (int t = lane; t < dp.nov; t += 32) S[yov + (int64_t)t * it.n] = y[dp.ovrow[t]];
		}
	}
}

__device__ __forceinline__ int dg_tiles(int n) { return (n + kDgTile - 1) / kDgTile; }

// The matrix to decompose (lower tiles), G or the kernel matrix, and with the latter X_te X_d^T.
__global__ void __launch_bounds__(kDgThreads) k_dg_gram(const DgItem *__restrict__ items, double *S, const DgParams dp) {
	extern __shared__ __align__(16) double dg_sm[];
	const DgItem it = items[blockIdx.y];
	const DgModel md = dp.mdl[it.model];
	const int tp = dg_tiles(it.p), low = tp * (tp + 1) / 2, d = md.d_n, n = it.n, te = md.te_n;
	int b = blockIdx.x, ti, tj;
	const bool first = b < low;
	if (first) {
		dg_lower(b, ti, tj);
	} else {
		b -= low;
		const int tt = dg_tiles(te);
		if (!it.dual || b >= tt * tp) return;
		ti = b % tt;
		tj = b / tt;
	}
	const int i0 = ti * kDgTile, j0 = tj * kDgTile;
	double acc[2][4][4];
	dg_zero(acc);
	int rows = it.p;
	if (!it.dual) {
		const DgOperand A = {S + it.xd, nullptr, d, n};
		dgemm_tile<true, true>(A, i0, A, j0, d, dg_sm, acc);
	} else {
		const DgOperand A = first ? DgOperand{S + it.xd, nullptr, d, d} : DgOperand{S + it.xte, nullptr, te, te};
		dgemm_tile<false, false>(A, i0, DgOperand{S + it.xd, nullptr, d, d}, j0, n, dg_sm, acc);
		if (!first) rows = te;
	}
	double *out = S + (first ? it.g : it.c);
	dg_each(acc, [&](int i, int j, double v) {
		if (i0 + i < rows && j0 + j < it.p) out[(int64_t)(j0 + j) * rows + i0 + i] = v;
	});
}

// W (d x p) or N (n x p), column-major, and E (te x p, row-major, scaled by the test weights).
__global__ void __launch_bounds__(kDgThreads) k_dg_project(const DgItem *__restrict__ items, double *S, const DgParams dp) {
	extern __shared__ __align__(16) double dg_sm[];
	const DgItem it = items[blockIdx.y];
	const DgModel md = dp.mdl[it.model];
	const int p = it.p, n = it.n, d = md.d_n, te = md.te_n;
	const int rows = it.dual ? n : d, tr = dg_tiles(rows), tp = dg_tiles(p), tt = dg_tiles(te);
	int b = blockIdx.x;
	const DgOperand V = {S + it.g, nullptr, p, p};
	double acc[2][4][4];
	dg_zero(acc);
	if (b < tr * tp) {
		const int i0 = (b % tr) * kDgTile, j0 = (b / tr) * kDgTile;
		if (it.dual) dgemm_tile<true, true>(DgOperand{S + it.xd, nullptr, d, n}, i0, V, j0, p, dg_sm, acc);
		else dgemm_tile<false, true>(DgOperand{S + it.xd, nullptr, d, d}, i0, V, j0, p, dg_sm, acc);
		double *out = S + (it.dual ? it.nv : it.c);
		dg_each(acc, [&](int i, int j, double v) {
			if (i0 + i < rows && j0 + j < p) out[(int64_t)(j0 + j) * rows + i0 + i] = v;
		});
		return;
	}
	b -= tr * tp;
	if (b >= tt * tp) return;
	const int i0 = (b % tt) * kDgTile, j0 = (b / tt) * kDgTile;
	dgemm_tile<false, true>(DgOperand{S + (it.dual ? it.c : it.xte), nullptr, te, te}, i0, V, j0, p, dg_sm, acc);
	double *E = S + it.e;
	const double *w = dp.tew + md.te_ofs;
	dg_each(acc, [&](int i, int j, double v) {
		if (i0 + i < te && j0 + j < p) E[(int64_t)(i0 + i) * p + j0 + j] = v * w[i0 + i];
	});
}

// The eigenvalues as squared column norms of W or N, a warp a column.
__global__ void __launch_bounds__(256) k_dg_lambda(const DgItem *__restrict__ items, double *S, const DgParams dp) {
	const DgItem it = items[blockIdx.y];
	const int rows = it.dual ? it.n : dp.mdl[it.model].d_n, lane = threadIdx.x & 31;
	const int r = (int)blockIdx.x * 8 + (threadIdx.x >> 5);
	if (r >= it.p) return;
	const double *col = S + (it.dual ? it.nv : it.c) + (int64_t)r * rows;
	double s = 0.0;
	for (int i = lane; i < rows; i += 32) s = fma(col[i], col[i], s);
	s = warp_sum(s);
	if (lane == 0) S[it.lam + r] = s;
}

// Q (p x n, column-major): W^T Y_d or U^T Y_d.
__global__ void __launch_bounds__(kDgThreads) k_dg_q(const DgItem *__restrict__ items, double *S, const DgParams dp) {
	extern __shared__ __align__(16) double dg_sm[];
	const DgItem it = items[blockIdx.y];
	const int p = it.p, n = it.n, d = dp.mdl[it.model].d_n, tp = dg_tiles(p), b = blockIdx.x;
	if (b >= tp * dg_tiles(n)) return;
	const int i0 = (b % tp) * kDgTile, j0 = (b / tp) * kDgTile;
	double acc[2][4][4];
	dg_zero(acc);
	dgemm_tile<true, true>(DgOperand{S + (it.dual ? it.g : it.c), nullptr, d, p}, i0, DgOperand{S + it.yd, nullptr, d, n}, j0, d,
	                       dg_sm, acc);
	double *Q = S + it.q;
	dg_each(acc, [&](int i, int j, double v) {
		if (i0 + i < p && j0 + j < n) Q[(int64_t)(j0 + j) * p + i0 + i] = v;
	});
}

// Whether component k is rounding noise: its singular value, the column norm of W or N, is below p eps of
// the largest, where a singular vector of a zero singular value ends up (its column of W is the sum of the
// others' rounding).  The bound is on the column norm: the same bound on the Gram matrix's eigenvalue
// drops true singular values up to sqrt(p eps) of the largest, which a small penalty still lets count (100
// rows, 100 columns of which 50 repeat the others to 1e-5, alpha = 1e-3: beta 3e-3 off; here 1.4e-10).
// NaN counts as a value.
__device__ __forceinline__ bool dg_noise(const double *lam, int p, int k) {
	const double r = p * Eps<double>::v();
	return lam[k] <= r * r * lam[0];
}

// 1 / (alpha + l_k); 0 for noise, so that alpha = 0 gives the pseudoinverse.
__device__ __forceinline__ double dg_coef(const double *lam, int p, int k, double alpha) {
	return dg_noise(lam, p, k) ? 0.0 : 1.0 / (alpha + lam[k]);
}

// Features of the searchlights of a one-model batch: the 64 largest singular values divided by the
// largest (zero-padded), then log n.
__global__ void __launch_bounds__(kFeatSv) k_dg_features(const DgItem *__restrict__ items, const DgSl *__restrict__ sls,
                                                         const double *__restrict__ S, float *__restrict__ feat) {
	const DgItem it = items[blockIdx.x];
	const double *lam = S + it.lam;
	float *f = feat + (int64_t)sls[blockIdx.x].s * (kFeatSv + 1);
	const int k = threadIdx.x;
	const double s1 = sqrt(lam[0]);
	f[k] = (k < it.p && s1 > 0.0 && !dg_noise(lam, it.p, k)) ? (float)(sqrt(lam[k]) / s1) : 0.0f;
	if (k == 0) f[kFeatSv] = logf((float)it.n);
}

// Position in the PC chunks: slice [k, min(k + 16, hi)) of chunk p (csrc/ha_ridge.c:187-210: chunk p
// is [npcs[p - 1], npcs[p]) clipped, possibly empty, and the chunks need not be monotone).
struct DgSlices {
	const int32_t *npcs;
	int n_npcs, K, p, k, hi;
	__device__ __forceinline__ void chunk() {
		while (p < n_npcs) {
			int r0, r1;
			pc_chunk(npcs, p, K, r0, r1);
			k = r0;
			hi = r1;
			if (k < hi) return;
			p++;
		}
	}
	__device__ __forceinline__ void start(const int32_t *npcs_, int n_, int K_) {
		npcs = npcs_; n_npcs = n_; K = K_; p = 0; k = hi = 0;
		chunk();
	}
	__device__ __forceinline__ void next() {
		k += kDgK;
		if (k >= hi) {
			p++;
			chunk();
		}
	}
};

// One tile (64 test rows x 64 targets) of one item at penalty a0 + blockIdx.y: the cumulative test
// predictions over the PC chunks in registers, E scaled by 1 / (alpha + l_k) as its fragments are read.
// Rows no other model tests give their squared error after every chunk (per-warp partials, summed in
// a fixed order by k_dg_cost); the others write their predictions.  The K slices run through the
// chunks without draining the pipeline between them.
__global__ void __launch_bounds__(kDgThreads) k_dg_eval(const DgItem *__restrict__ items, const DgSl *__restrict__ sls,
                                                        double *S, const DgParams dp, int a0) {
	extern __shared__ __align__(16) double dg_sm[];
	__shared__ double cv[kEigMaxP];
	const DgItem it = items[blockIdx.z];
	const DgModel md = dp.mdl[it.model];
	const int p = it.p, n = it.n, te = md.te_n, tt = dg_tiles(te), tn = dg_tiles(n);
	if ((int)blockIdx.x >= tt * tn) return;
	const int i0 = ((int)blockIdx.x % tt) * kDgTile, j0 = ((int)blockIdx.x / tt) * kDgTile, a = a0 + (int)blockIdx.y;
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	const int g = lane >> 2, t = lane & 3, wm = 32 * (warp & 1), wn = 32 * (warp >> 1);
	const double *lam = S + it.lam;
	const double alpha = dp.alphas[a];
	const int K = p;  // at most min(rows, n), where the reference clips: the components past p are zero
	for (int k = tid; k < K; k += kDgThreads) cv[k] = dg_coef(lam, p, k, alpha);
	const DgSl sl = sls[it.sl];
	double acc[2][4][4];
	const double *Yt = S + it.yte;
#pragma unroll
	for (int u = 0; u < 2; u++)
#pragma unroll
		for (int v = 0; v < 4; v++)
#pragma unroll
			for (int e = 0; e < 4; e++) {
				const int i = i0 + wm + 16 * u + g + 8 * (e >> 1), j = j0 + wn + 8 * v + 2 * t + (e & 1);
				acc[u][v][e] = (i < md.te1 && j < n) ? -Yt[(int64_t)j * te + i] : 0.0;
			}
	const double *E = S + it.e, *Q = S + it.q;
	DgLoader<true> la, lb;
	la.init(DgOperand{E, nullptr, p, te}, i0, tid);
	lb.init(DgOperand{Q, nullptr, p, n}, j0, tid);
	DgSlices ld, cp;
	ld.start(dp.npcs, dp.n_npcs, K);
	int filled = 0;
	auto fill = [&]() {
		if (ld.p < dp.n_npcs) {
			double *st = dg_sm + (filled % kDgStages) * 2 * kDgOperand;
			la.load(st, ld.k, ld.hi, E);
			lb.load(st + kDgOperand, ld.k, ld.hi, E);
			ld.next();
		}
		filled++;
		asm volatile("cp.async.commit_group;" ::: "memory");
	};
#pragma unroll
	for (int s = 0; s < kDgStages - 1; s++) fill();
	cp.start(dp.npcs, dp.n_npcs, K);
	double *part = S + sl.part + (int64_t)a * dp.n_npcs * sl.nparts + it.part0 + 4 * (int)blockIdx.x + warp;
	const bool active = dg_active(i0, te, j0, n);
	int emitted = 0;
	auto emit = [&](int upto) {  // grid points [emitted, upto) of this penalty have these predictions
		if (emitted >= upto) return;
		double ss = 0.0;
#pragma unroll
		for (int u = 0; u < 2; u++)
#pragma unroll
			for (int v = 0; v < 4; v++)
#pragma unroll
				for (int e = 0; e < 4; e++) {
					const int i = i0 + wm + 16 * u + g + 8 * (e >> 1);
					if (i < md.te1) ss = fma(acc[u][v][e], acc[u][v][e], ss);  // columns past n hold zeros
				}
		ss = warp_sum(ss);
		for (; emitted < upto; emitted++) {
			if (lane == 0) part[(int64_t)emitted * sl.nparts] = ss;
			if (i0 + kDgTile <= md.te1) continue;
			double *P = S + sl.pov + (((int64_t)blockIdx.y * dp.n_npcs + emitted) * dp.entries + md.entry0) * n;
#pragma unroll
			for (int u = 0; u < 2; u++)
#pragma unroll
				for (int v = 0; v < 4; v++)
#pragma unroll
					for (int e = 0; e < 4; e++) {
						const int i = i0 + wm + 16 * u + g + 8 * (e >> 1), j = j0 + wn + 8 * v + 2 * t + (e & 1);
						if (i >= md.te1 && i < te && j < n) P[(int64_t)(i - md.te1) * n + j] = acc[u][v][e];
					}
		}
	};
	for (int s = 0; cp.p < dp.n_npcs; s++) {
		emit(cp.p);  // the chunks before this slice's are complete
		asm volatile("cp.async.wait_group %0;" ::"n"(kDgStages - 2) : "memory");
		__syncthreads();
		fill();
		const double *as = dg_sm + (s % kDgStages) * 2 * kDgOperand, *bs = as + kDgOperand;
		if (active)
#pragma unroll
		for (int kk = 0; kk < kDgK; kk += 8) {
			double x[2][4], y[4][2];
			// slots past the chunk's end hold zeros in both operands; their scale only has to be finite
			const double c0 = cp.k + kk + t < cp.hi ? cv[cp.k + kk + t] : 0.0;
			const double c1 = cp.k + kk + t + 4 < cp.hi ? cv[cp.k + kk + t + 4] : 0.0;
#pragma unroll
			for (int u = 0; u < 2; u++)
#pragma unroll
				for (int e = 0; e < 4; e++)
					x[u][e] = dg_frag<true>(as, wm + 16 * u + g + 8 * (e & 1), kk + t + 4 * (e >> 1)) * (e >> 1 ? c1 : c0);
#pragma unroll
			for (int v = 0; v < 4; v++)
#pragma unroll
				for (int e = 0; e < 2; e++) y[v][e] = dg_frag<true>(bs, wn + 8 * v + g, kk + t + 4 * e);
#pragma unroll
			for (int u = 0; u < 2; u++)
#pragma unroll
				for (int v = 0; v < 4; v++) dg_mma(acc[u][v], x[u], y[v]);
		}
		cp.next();
	}
	asm volatile("cp.async.wait_group 0;" ::: "memory");
	emit(dp.n_npcs);
}

// Squared error of kDgRows several-model rows (blockIdx.z) of one searchlight (blockIdx.y) at one grid point
// (penalty a0 + blockIdx.x / n_npcs), a warp a row: one more partial of the grid point.
constexpr int kDgRows = 16;
__global__ void __launch_bounds__(256) k_dg_cost(const DgSl *__restrict__ sls, double *S, const DgParams dp, int a0) {
	__shared__ double red[32];
	const DgSl sl = sls[blockIdx.y];
	const int n = sl.n, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	const double *P = S + sl.pov + (int64_t)blockIdx.x * dp.entries * n, *Yov = S + sl.yov;
	double s = 0.0;
	for (int u = kDgRows * blockIdx.z + warp; u < min(kDgRows * ((int)blockIdx.z + 1), dp.nov); u += 8) {
		const int e0 = dp.ovptr[u], e1 = dp.ovptr[u + 1];
		const double *p0 = P + (int64_t)dp.ovent[e0] * n, *p1 = P + (int64_t)dp.ovent[e0 + 1] * n;  // at least two
		const double *y = Yov + (int64_t)u * n;
		if (e1 - e0 == 2) {
#pragma unroll 4
			for (int j = lane; j < n; j += 32) {
				const double x = p0[j] + p1[j] - y[j];
				s = fma(x, x, s);
			}
		} else {
			for (int j = lane; j < n; j += 32) {
				double x = p0[j] + p1[j];
				for (int e = e0 + 2; e < e1; e++) x += P[(int64_t)dp.ovent[e] * n + j];
				x -= y[j];
				s = fma(x, x, s);
			}
		}
	}
	s = grid_block_sum(s, red);
	if (threadIdx.x == 0)
		S[sl.part + ((int64_t)a0 * dp.n_npcs + blockIdx.x) * sl.nparts + sl.nparts - gridDim.z + blockIdx.z] = s;
}

// The grid points' costs (their partials in order, a warp a grid point), the winner (first minimum of the
// summed cost, csrc/ha_ridge.c:322-327) and the cost row with the untested rows' squared targets added
// (their prediction is zero, csrc/ha_ridge.c:297-319).
__global__ void __launch_bounds__(256) k_dg_best(const DgSl *__restrict__ sls, const int32_t *__restrict__ sl_idx,
                                                 const double *__restrict__ Y, double *S, const DgParams dp,
                                                 int32_t *__restrict__ best_out,
                                                 double *__restrict__ cost_out) {
	__shared__ double red[32];
	const DgSl sl = sls[blockIdx.x];
	const int grid = dp.n_alphas * dp.n_npcs;
	double *cost = S + sl.cost;
	for (int gi = threadIdx.x >> 5; gi < grid; gi += blockDim.x >> 5) {
		const double *part = S + sl.part + (int64_t)gi * sl.nparts;
		double c = 0.0;
		for (int i = threadIdx.x & 31; i < sl.nparts; i += 32) c += part[i];
		c = warp_sum(c);
		if ((threadIdx.x & 31) == 0) cost[gi] = c;
	}
	double yc = 0.0;
	for (int64_t e = threadIdx.x; e < (int64_t)dp.n_untested * sl.n; e += blockDim.x) {
		const int j = (int)(e / dp.n_untested), t = (int)(e - (int64_t)j * dp.n_untested);
		const double y = Y[(int64_t)sl_idx[sl.sofs + j] * dp.nt + dp.untested[t]];
		yc = fma(y, y, yc);
	}
	yc = grid_block_sum(yc, red);
	if (threadIdx.x == 0) {
		int b = 0;
		for (int gi = 1; gi < grid; gi++)
			if (cost[gi] < cost[b]) b = gi;
		best_out[sl.s] = b;
	}
	if (cost_out)
		for (int gi = threadIdx.x; gi < grid; gi += blockDim.x) cost_out[(int64_t)sl.s * grid + gi] = cost[gi] + yc;
}

// One tile of the winner's model-averaged beta, written in the T layout (row-major for CSR output,
// column-major for CSC): the sum over models of N diag(m_k / (alpha + l_k)) Q, m_k the number of PC
// chunks up to the winner's that hold component k.  With prob, only searchlights whose proposal `best`
// has at least that probability (one model: the fit at the proposed grid point).
__global__ void __launch_bounds__(kDgThreads) k_dg_beta(const DgItem *__restrict__ items, const DgSl *__restrict__ sls,
                                                        const double *__restrict__ S, const DgParams dp,
                                                        const int32_t *__restrict__ best, const float *__restrict__ prob,
                                                        float min_prob, double *__restrict__ Bout, int t_rowmajor) {
	extern __shared__ __align__(16) double dg_sm[];
	__shared__ double cv[kEigMaxP];
	__shared__ int s_top;
	const DgSl sl = sls[blockIdx.y];
	const int n = sl.n, tn = dg_tiles(n), tid = threadIdx.x;
	if ((int)blockIdx.x >= tn * tn || (prob && prob[sl.s] < min_prob)) return;
	const int i0 = ((int)blockIdx.x % tn) * kDgTile, j0 = ((int)blockIdx.x / tn) * kDgTile;
	const int b = best[sl.s], ba = b / dp.n_npcs, bp = b - ba * dp.n_npcs;
	const double alpha = dp.alphas[ba];
	double sum[2][4][4];
	dg_zero(sum);
	for (int mo = 0; mo < dp.models; mo++) {
		const DgItem it = items[sl.item0 + mo];
		const double *lam = S + it.lam;
		const int K = it.p;
		__syncthreads();
		if (tid == 0) s_top = 0;
		__syncthreads();
		for (int k = tid; k < K; k += kDgThreads) {
			int mult = 0;
			for (int p = 0; p <= bp; p++) {
				int r0, r1;
				pc_chunk(dp.npcs, p, K, r0, r1);
				mult += (k >= r0 && k < r1) ? 1 : 0;
			}
			cv[k] = mult ? (double)mult * dg_coef(lam, it.p, k, alpha) : 0.0;
			if (mult) atomicMax(&s_top, k + 1);
		}
		__syncthreads();
		const int top = s_top;
		DgLoader<false> la;
		DgLoader<true> lb;
		la.init(DgOperand{S + it.nv, nullptr, n, n}, i0, tid);
		lb.init(DgOperand{S + it.q, nullptr, it.p, n}, j0, tid);
		dgemm_core(la, lb, top, S + it.q, dg_sm, sum, dg_active(i0, n, j0, n), cv);
	}
	double *Bo = Bout + sl.tofs;
	const int64_t ti = t_rowmajor ? n : 1, tj = t_rowmajor ? 1 : n;
	dg_each(sum, [&](int i, int j, double v) {
		if (i0 + i < n && j0 + j < n) Bo[(int64_t)(i0 + i) * ti + (int64_t)(j0 + j) * tj] = v / dp.models;
	});
}

}  // namespace hab200
