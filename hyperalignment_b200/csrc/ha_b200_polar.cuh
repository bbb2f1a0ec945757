// ha_b200_polar.cuh -- batched float64 polar factors by the scaled Newton-Schulz iteration
//     X_0 = B / u,   X_{k+1} = X_k (c1 I + c3 X_k^T X_k),   u >= sigma_max(B),
// every product a set of 64 x 64 tiles on the float64 tensor cores (one CTA a tile, so the whole
// batch fills the chip; the one-sided Jacobi polar runs one CTA a matrix and is bound by its
// shared-memory rotations).  The schedule is the float32 solver's (ns_schedule): about 16 iterations of
// 3 n^3 multiply-adds: 8 ms for 256 matrices of order 100-300, where the Jacobi polar took 230.  A matrix ends after one more update once ||X^T X - I||_F / sqrt(n) is below 1e-8
// on a plain step (the step squares it); one that stalls (singular values that stay zero) or
// reaches the iteration limit is flagged kFlagIllCond for the Jacobi solve.
#pragma once

#include "ha_b200_dgemm.cuh"

namespace hab200 {

struct PolarWork {
	int64_t b;       // B (n x n, column-major) in the launch's B base
	int64_t x, x2, g;  // two iterates and the Gram product in the scratch base
	int64_t t;       // T (float, column-major) in the T base
	int32_t n, slot;
	int32_t part;    // first residual partial of the matrix (one per lower tile)
	int32_t pad_;
};

struct PolarTile {
	int32_t w, t;  // matrix, tile (lower tiles first)
};

struct PolarState {
	int32_t done, plain, conv, pad_;
	double res;
};

struct PolarArgs {
	const PolarWork *work;
	const PolarTile *tiles;
	const double *B;
	double *S;          // scratch
	float *T;
	double *part;
	const PolarState *in;
	PolarState *out;
	int32_t *left;      // matrices not finished after this update
	double c1, c3;
	int plain, last, odd;  // odd: the iterate is in x2
};

constexpr double kPolarTol = 1e-8;

__global__ void __launch_bounds__(256) k_polar_init(const PolarArgs a) {
	const PolarWork w = a.work[blockIdx.x];
	const int n = w.n, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	const double *B = a.B + w.b;
	__shared__ double s_red[3][8];
	double fro = 0.0, cmax = 0.0, rmax = 0.0;
	for (int c = warp; c < n; c += 8) {  // column sums of |B|
		double s = 0.0;
		for (int r = lane; r < n; r += 32) {
			const double x = B[(int64_t)c * n + r];
			fro = fma(x, x, fro);
			s += fabs(x);
		}
		cmax = fmax(cmax, warp_sum(s));
	}
	for (int r = threadIdx.x; r < n; r += blockDim.x) {  // row sums
		double s = 0.0;
		for (int c = 0; c < n; c++) s += fabs(B[(int64_t)c * n + r]);
		rmax = fmax(rmax, s);
	}
	fro = warp_sum(fro);
	for (int o = 16; o > 0; o >>= 1) rmax = fmax(rmax, __shfl_xor_sync(0xffffffffu, rmax, o));
	if (lane == 0) {
		s_red[0][warp] = fro;
		s_red[1][warp] = cmax;
		s_red[2][warp] = rmax;
	}
	__syncthreads();
	fro = cmax = rmax = 0.0;
	for (int i = 0; i < 8; i++) {
		fro += s_red[0][i];
		cmax = fmax(cmax, s_red[1][i]);
		rmax = fmax(rmax, s_red[2][i]);
	}
	double u = fmin(sqrt(fro), sqrt(cmax) * sqrt(rmax));
	if (!(u > 0.0)) u = 1.0;  // zero matrix: the iterate stays zero and the matrix is flagged
	const double inv = 1.0 / (u * (1.0 + 1e-12));
	for (int64_t e = threadIdx.x; e < (int64_t)n * n; e += blockDim.x) a.S[w.x + e] = B[e] * inv;
	if (threadIdx.x == 0) a.out[blockIdx.x] = PolarState{0, 0, 0, 0, 0.0};
}

// G = X^T X (lower tiles, mirrored) and the tile's part of ||G - I||_F^2.
__global__ void __launch_bounds__(kDgThreads) k_polar_gram(const PolarArgs a) {
	extern __shared__ __align__(16) double dg_sm[];
	__shared__ double red[kDgThreads / 32];
	const PolarTile tl = a.tiles[blockIdx.x];
	if (a.in[tl.w].done) return;
	const PolarWork w = a.work[tl.w];
	const int n = w.n;
	int ti, tj;
	dg_lower(tl.t, ti, tj);
	const int i0 = ti * kDgTile, j0 = tj * kDgTile;
	const DgOperand X = {a.S + (a.odd ? w.x2 : w.x), nullptr, n, n};
	double acc[2][4][4];
	dg_zero(acc);
	dgemm_tile<true, true>(X, i0, X, j0, n, dg_sm, acc);
	double *G = a.S + w.g;
	double ss = 0.0;
	dg_each(acc, [&](int i, int j, double v) {
		const int r = i0 + i, c = j0 + j;
		if (r >= n || c >= n) return;
		G[(int64_t)c * n + r] = v;
		if (ti != tj) G[(int64_t)r * n + c] = v;
		const double d = v - (r == c ? 1.0 : 0.0);
		ss = fma(d, d, ss);
	});
	ss = warp_sum(ss);
	if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
	__syncthreads();
	if (threadIdx.x == 0) {
		double s = 0.0;
		for (int i = 0; i < kDgThreads / 32; i++) s += red[i];
		a.part[w.part + tl.t] = ti == tj ? s : 2.0 * s;
	}
}

// X <- X (c1 I + c3 G), or T for the last update (decided alike by every tile of the matrix).
__global__ void __launch_bounds__(kDgThreads) k_polar_update(const PolarArgs a) {
	extern __shared__ __align__(16) double dg_sm[];
	const PolarTile tl = a.tiles[blockIdx.x];
	const PolarState st = a.in[tl.w];
	if (st.done) {
		if (tl.t == 0 && threadIdx.x == 0) a.out[tl.w] = st;
		return;
	}
	const PolarWork w = a.work[tl.w];
	const int n = w.n, T = (n + kDgTile - 1) / kDgTile, low = T * (T + 1) / 2;
	double ss = 0.0;
	for (int i = 0; i < low; i++) ss += a.part[w.part + i];
	const double res = sqrt(ss / n);
	const bool conv = a.plain && res < kPolarTol;
	// plain steps that leave the residual as it is: some singular values stay zero
	const bool stalled = !conv && a.plain && st.plain && !(fabs(res - st.res) > 1e-13 * res);
	const bool fin = conv || stalled || a.last;
	if (tl.t == 0 && threadIdx.x == 0) {
		a.out[tl.w] = PolarState{fin ? 1 : 0, a.plain, conv ? 1 : 0, 0, res};
		if (!fin) atomicAdd(a.left, 1);
	}
	const int i0 = (tl.t % T) * kDgTile, j0 = (tl.t / T) * kDgTile;
	const double *X = a.S + (a.odd ? w.x2 : w.x);
	double acc[2][4][4];
	dg_zero(acc);
	dgemm_tile<false, true>(DgOperand{X, nullptr, n, n}, i0, DgOperand{a.S + w.g, nullptr, n, n}, j0, n, dg_sm, acc);
	double *Xn = a.S + (a.odd ? w.x : w.x2);
	float *Tm = a.T + w.t;
	dg_each(acc, [&](int i, int j, double v) {
		const int r = i0 + i, c = j0 + j;
		if (r >= n || c >= n) return;
		const int64_t e = (int64_t)c * n + r;
		const double x = a.c1 * X[e] + a.c3 * v;
		if (fin) Tm[e] = (float)x;
		else Xn[e] = x;
	});
}

__global__ void k_polar_finish(const PolarWork *__restrict__ work, int n, const PolarState *__restrict__ st,
                               SlStats *__restrict__ stats) {
	const int q = blockIdx.x * blockDim.x + threadIdx.x;
	if (q < n) stats[work[q].slot].flags = st[q].conv ? kFlagFP64 : kFlagIllCond;
}

}  // namespace hab200
