// ha_b200_eig.cuh -- batched float64 eigen decomposition of symmetric matrices (order 1..512).
//
// One-sided Jacobi on a factor of the matrix needs about ten sweeps of 4 p^3 operations whose
// every rotation is two passes over two columns in shared memory, a barrier per round: measured
// 31 ms of one SM per matrix of order 275.  Here: Householder tridiagonalisation (4/3 p^3, bound by
// reading the trailing block once per column through L2), the explicit basis Q (4/3 p^3 on the
// float64 tensor cores), the implicit QL iteration on the tridiagonal matrix (serial, one warp per
// matrix, thousands of matrices at once), and its recorded rotations applied to the rows of Q, a
// thread a row and eight sweeps at a time.  256 matrices of order 400: 41 ms (tridiagonalisation and
// basis 14.7, QL 16.8, rotations 9.8) against about 250 ms of Jacobi sweeps.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "ha_b200_dgemm.cuh"

namespace hab200 {

constexpr int kEigMaxP = 512;
constexpr int kEigNb = 16;       // columns per reduction panel and per block reflector
constexpr int kEigThreads = 256;
constexpr int kEigSweeps = 8;    // QL sweeps applied together
constexpr int kEigRounds = 2;    // QL launches; the second finishes what the first had no room for

// One matrix.  A (p x p, the lower triangle is read, column-major) is overwritten by the eigenvectors, columns
// in decreasing order of the eigenvalues; Q is p x p scratch; lam receives the eigenvalues, each with
// an error of a few eps lambda_max (those of a singular matrix are rounding of either sign).  No
// eigenvector is dropped for it: of X^T X, a singular value of X down to sqrt(eps) of the largest ends
// there, and its component still counts for a ridge fit at a small penalty.
struct EigWork {
	int64_t a, q, s, lam;  // element offsets from the launch's four base pointers
	int32_t p, pad_;
};

// Scratch of one matrix from EigWork::s, in float64 elements.
struct EigScratch {
	int64_t d, e, tau, vv, rank, state, sweep, rot, total;
	int cap;  // sweeps per round
	__host__ __device__ static EigScratch make(int p) {
		EigScratch L;
		L.cap = 2 * p + 16;
		int64_t o = 0;
		L.d = o; o += p;
		L.e = o; o += p;
		L.tau = o; o += p;
		L.vv = o; o += (int64_t)p * kEigNb;  // V^T v_j of column j's panel
		L.rank = o; o += p;
		L.state = o; o += 4;
		L.sweep = o; o += L.cap;              // int2 (first, one past last) rotation of each sweep
		o = (o + 1) & ~(int64_t)1;
		L.rot = o; o += (int64_t)L.cap * p * 2;  // double2 (c, s) per sweep and column
		L.total = (o + 3) & ~(int64_t)3;
		return L;
	}
};

struct EigState {
	int32_t next;    // first eigenvalue not yet found
	int32_t sweeps;  // sweeps recorded in the last round
	int32_t done;    // round (1, 2) in which the iteration finished, 0: not yet
	int32_t bad;     // ended without converging
	double scale;    // the tridiagonal matrix holds T / scale
};

__host__ __device__ __forceinline__ int eig_ld(int p) { return ((p + 22) & ~15) + 4; }
__host__ __device__ __forceinline__ size_t eig_tridiag_smem(int p) {
	return ((size_t)(2 * kEigNb + 1 + kEigThreads / 32) * eig_ld(p) + 8 * 16 * 10 + 16 * 17 + 64) * sizeof(double);
}

__device__ __forceinline__ double eig_block_sum(double v, double *red) {
	v = warp_sum(v);
	if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
	__syncthreads();
	double t = 0.0;
#pragma unroll
	for (int i = 0; i < kEigThreads / 32; i++) t += red[i];
	return t;
}

// Tridiagonalisation A = Q T Q^T and the explicit Q, one CTA per matrix, p <= 32 RK.  Panels of 16
// columns: inside a panel the lower triangle of the trailing block is read once per column (the
// product A v; the panel's earlier rank-2 updates are applied to the vectors), after it the triangle
// takes one rank-32 update on the float64 tensor cores.  The panel (V and W, row index fastest)
// stays in shared memory.  In the product a warp takes whole columns and a lane the rows
// lane + 32 k: v and the lane's share of the transposed half's sums stay in registers, so an element
// costs one load and two multiply-adds and no shared memory.
template <int RK>
__global__ void __launch_bounds__(kEigThreads, RK <= 8 ? 2 : 1) k_eig_tridiag(const EigWork *__restrict__ work, double *Ab, double *Qb,
                                                                double *Sb) {
	extern __shared__ __align__(16) double eg_sm[];
	const EigWork w = work[blockIdx.x];
	const int p = w.p, ld = eig_ld(p);
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
	constexpr int kWarps = kEigThreads / 32;
	double *A = Ab + w.a, *Q = Qb + w.q;
	const EigScratch L = EigScratch::make(p);
	double *sd = Sb + w.s + L.d, *se = Sb + w.s + L.e, *stau = Sb + w.s + L.tau, *svv = Sb + w.s + L.vv;
	double *V = eg_sm, *W = V + kEigNb * ld, *col = W + kEigNb * ld;
	double *yb = col + ld;                  // per warp: the transposed half's sums
	double *wb = yb + kWarps * ld;          // 16 x 8 per warp, leading dimension 10
	double *Tm = wb + kWarps * 16 * 10;     // 16 x 16, leading dimension 17
	double *sml = Tm + 16 * 17;             // the panel's dot products: V^T v, W^T v
	double *red = sml + 32, *red2 = red + 8;
	for (int j0 = 0; j0 < p - 1; j0 += kEigNb) {
		const int nbk = min(kEigNb, p - 1 - j0);
		for (int e = tid; e < 2 * kEigNb * ld; e += kEigThreads) V[e] = 0.0;  // V and W
		constexpr int kColElems = (32 * RK + kEigThreads - 1) / kEigThreads;
		double nxt[kColElems];
#pragma unroll
		for (int x2 = 0; x2 < kColElems; x2++) {
			const int r = tid + kEigThreads * x2;
			nxt[x2] = (r >= j0 && r < p) ? A[(int64_t)j0 * p + r] : 0.0;
		}
		__syncthreads();
		for (int i = 0; i < nbk; i++) {
			const int j = j0 + i;
			// column j with the panel's earlier updates, and the norm below its first subdiagonal entry
			double ss = 0.0;
#pragma unroll
			for (int x2 = 0; x2 < kColElems; x2++) {
				const int r = tid + kEigThreads * x2;
				if (r < j || r >= p) continue;
				double x = nxt[x2];
				for (int q = 0; q < i; q++) x -= V[q * ld + r] * W[q * ld + j] + W[q * ld + r] * V[q * ld + j];
				col[r] = x;
				if (r > j + 1) ss += x * x;
			}
			// the next column of the panel is on its way while this one is worked on
			if (i + 1 < nbk) {
#pragma unroll
				for (int x2 = 0; x2 < kColElems; x2++) {
					const int r = tid + kEigThreads * x2;
					nxt[x2] = (r > j && r < p) ? A[(int64_t)(j + 1) * p + r] : 0.0;
				}
			}
			ss = eig_block_sum(ss, red);
			// reflector I - tau v v^T (v_1 = 1) that maps the column below the diagonal to beta e_1
			const double alpha = col[j + 1];
			double beta = alpha, tau = 0.0, scl = 0.0;
			if (ss > 0.0) {
				beta = -copysign(sqrt(alpha * alpha + ss), alpha);
				tau = (beta - alpha) / beta;
				scl = 1.0 / (alpha - beta);
			}
			for (int r = j + 1 + tid; r < p; r += kEigThreads) {
				const double v = r == j + 1 ? 1.0 : col[r] * scl;
				V[i * ld + r] = v;
				A[(int64_t)j * p + r] = v;
			}
			if (tid == 0) {
				sd[j] = col[j];
				se[j] = beta;
				stau[j] = tau;
			}
			__syncthreads();
			// y = A v over the trailing block, a warp four columns at a time; the panel's dot products
			const double *v = V + i * ld;
			{
				// NC columns' elements are all in flight together
				constexpr int NC = RK <= 8 ? 2 : 4;
				double vr[RK], ya[RK];
#pragma unroll
				for (int k = 0; k < RK; k++) {
					vr[k] = 32 * k + lane < p ? v[32 * k + lane] : 0.0;
					ya[k] = 0.0;
				}
				for (int c0 = j + 1 + warp; c0 < p; c0 += NC * kWarps) {
					double s4[NC], el[NC][RK];
#pragma unroll
					for (int x = 0; x < NC; x++) {
						const int c = c0 + kWarps * x;
						const double *a = A + (int64_t)min(c, p - 1) * p + lane;
#pragma unroll
						for (int k = 0; k < RK; k++) el[x][k] = (32 * k + lane >= c && 32 * k + lane < p) ? a[32 * k] : 0.0;
					}
#pragma unroll
					for (int x = 0; x < NC; x++) {
						const int c = c0 + kWarps * x;
						const double vc = c < p ? v[c] : 0.0;
						s4[x] = 0.0;
#pragma unroll
						for (int k = 0; k < RK; k++) {
							s4[x] = fma(el[x][k], vr[k], s4[x]);
							ya[k] = fma(32 * k + lane != c ? el[x][k] : 0.0, vc, ya[k]);
						}
					}
					const double s = pair_sums<double, NC>(s4, lane);
					const int c = c0 + kWarps * (lane / (32 / NC));
					if ((lane & (32 / NC - 1)) == 0 && c < p) W[i * ld + c] = s;
				}
#pragma unroll
				for (int k = 0; k < RK; k++)
					if (32 * k + lane < p) yb[warp * ld + 32 * k + lane] = ya[k];
			}
			for (int q = warp; q < 2 * i; q += kWarps) {
				const double *u = q < i ? V + q * ld : W + (q - i) * ld;
				double s = 0.0;
				for (int r = j + 1 + lane; r < p; r += 32) s = fma(u[r], v[r], s);
				s = warp_sum(s);
				if (lane == 0) sml[q < i ? q : kEigNb + q - i] = s;
			}
			__syncthreads();
			if (tid < i) svv[(int64_t)j * kEigNb + tid] = sml[tid];
			// w = tau (y - V (W^T v) - W (V^T v)), then w -= tau (w^T v) / 2 v
			double dot = 0.0;
			for (int c = j + 1 + tid; c < p; c += kEigThreads) {
				double y = W[i * ld + c];
#pragma unroll
				for (int q = 0; q < kWarps; q++) y += yb[q * ld + c];
				for (int q = 0; q < i; q++) y -= V[q * ld + c] * sml[kEigNb + q] + W[q * ld + c] * sml[q];
				y *= tau;
				W[i * ld + c] = y;
				dot = fma(y, v[c], dot);
			}
			dot = eig_block_sum(dot, red2);
			for (int c = j + 1 + tid; c < p; c += kEigThreads) W[i * ld + c] -= 0.5 * tau * dot * v[c];
			__syncthreads();
		}
		// A22 -= V W^T + W V^T, the lower 32 x 32 blocks, a warp a block
		const int t0 = j0 + nbk, nt32 = (p - t0 + 31) >> 5;
		for (int b = warp; b < nt32 * nt32; b += kWarps) {
			const int r0 = t0 + 32 * (b % nt32), c0 = t0 + 32 * (b / nt32);
			if (r0 < c0) continue;
			double acc[2][4][4];
			dg_zero(acc);
#pragma unroll
			for (int ks = 0; ks < 4; ks++) {
				const double *L0 = (ks < 2 ? V : W) + (ks & 1) * 8 * ld, *R0 = (ks < 2 ? W : V) + (ks & 1) * 8 * ld;
				double a[2][4], bb[4][2];
#pragma unroll
				for (int u = 0; u < 2; u++)
#pragma unroll
					for (int e = 0; e < 4; e++) a[u][e] = L0[(t + 4 * (e >> 1)) * ld + min(r0 + 16 * u + g + 8 * (e & 1), p - 1)];
#pragma unroll
				for (int x = 0; x < 4; x++)
#pragma unroll
					for (int e = 0; e < 2; e++) bb[x][e] = R0[(t + 4 * e) * ld + min(c0 + 8 * x + g, p - 1)];
#pragma unroll
				for (int u = 0; u < 2; u++)
#pragma unroll
					for (int x = 0; x < 4; x++) dg_mma(acc[u][x], a[u], bb[x]);
			}
			// every element is read before the first is written
			double old[2][4][4];
#pragma unroll
			for (int u = 0; u < 2; u++)
#pragma unroll
				for (int x = 0; x < 4; x++)
#pragma unroll
					for (int e = 0; e < 4; e++) {
						const int r = r0 + 16 * u + g + 8 * (e >> 1), c = c0 + 8 * x + 2 * t + (e & 1);
						old[u][x][e] = (r < p && c < p) ? A[(int64_t)c * p + r] : 0.0;
					}
#pragma unroll
			for (int u = 0; u < 2; u++)
#pragma unroll
				for (int x = 0; x < 4; x++)
#pragma unroll
					for (int e = 0; e < 4; e++) {
						const int r = r0 + 16 * u + g + 8 * (e >> 1), c = c0 + 8 * x + 2 * t + (e & 1);
						if (r < p && c < p) A[(int64_t)c * p + r] = old[u][x][e] - acc[u][x][e];
					}
		}
		__syncthreads();
	}
	if (tid == 0) {
		sd[p - 1] = A[(int64_t)(p - 1) * p + p - 1];
		se[p - 1] = 0.0;
		*reinterpret_cast<EigState *>(Sb + w.s + L.state) = EigState{0, 0, 0, 0, 0.0};
	}
	// Q = H_0 H_1 ..: block reflectors I - V T V^T applied to the identity, the last block first
	for (int64_t e = tid; e < (int64_t)p * p; e += kEigThreads) {
		const int c = (int)(e / p), r = (int)(e - (int64_t)c * p);
		Q[e] = r == c ? 1.0 : 0.0;
	}
	for (int j0 = ((p - 2) / kEigNb) * kEigNb; j0 >= 0 && p > 1; j0 -= kEigNb) {
		const int nbk = min(kEigNb, p - 1 - j0);
		__syncthreads();
		for (int e = tid; e < kEigNb * ld; e += kEigThreads) {
			const int q = e / ld, r = e - q * ld;
			V[e] = (q < nbk && r > j0 + q && r < p) ? A[(int64_t)(j0 + q) * p + r] : 0.0;
		}
		if (warp == 0) {
			for (int e = lane; e < 16 * 17; e += 32) Tm[e] = 0.0;
			__syncwarp();
			for (int i = 0; i < nbk; i++) {
				const double tau = stau[j0 + i];
				double s = 0.0;
				if (lane < i)
					for (int k = lane; k < i; k++) s = fma(Tm[lane * 17 + k], svv[(int64_t)(j0 + i) * kEigNb + k], s);
				if (lane < i) Tm[lane * 17 + i] = -tau * s;
				if (lane == i) Tm[i * 17 + i] = tau;
				__syncwarp();
			}
		}
		__syncthreads();
		double *wq = wb + warp * 16 * 10;
		for (int c0 = j0 + 1 + 8 * warp; c0 < p; c0 += 8 * kWarps) {
			const double *qc = Q + (int64_t)min(c0 + g, p - 1) * p;
			double acc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 4
			for (int r = j0 + 1; r < p; r += 8) {
				const double a[4] = {V[g * ld + r + t], V[(g + 8) * ld + r + t], V[g * ld + r + t + 4], V[(g + 8) * ld + r + t + 4]};
				const double b[2] = {qc[min(r + t, p - 1)], qc[min(r + t + 4, p - 1)]};
				dg_mma(acc, a, b);
			}
			__syncwarp();
#pragma unroll
			for (int e = 0; e < 4; e++) wq[(g + 8 * (e >> 1)) * 10 + 2 * t + (e & 1)] = acc[e];
			__syncwarp();
			double a2[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
			for (int k = 0; k < 16; k += 8) {
				const double a[4] = {Tm[g * 17 + k + t], Tm[(g + 8) * 17 + k + t], Tm[g * 17 + k + t + 4], Tm[(g + 8) * 17 + k + t + 4]};
				const double b[2] = {wq[(k + t) * 10 + g], wq[(k + t + 4) * 10 + g]};
				dg_mma(a2, a, b);
			}
			__syncwarp();
#pragma unroll
			for (int e = 0; e < 4; e++) wq[(g + 8 * (e >> 1)) * 10 + 2 * t + (e & 1)] = a2[e];
			__syncwarp();
			const double b0[2] = {wq[t * 10 + g], wq[(t + 4) * 10 + g]};
			const double b1[2] = {wq[(t + 8) * 10 + g], wq[(t + 12) * 10 + g]};
			// four 16-row pieces at a time, read before the first is written
			for (int rq = j0 + 1; rq < p; rq += 64) {
				double old[4][4];
#pragma unroll
				for (int x = 0; x < 4; x++)
#pragma unroll
					for (int e = 0; e < 4; e++) {
						const int rr = rq + 16 * x + g + 8 * (e >> 1), cc = c0 + 2 * t + (e & 1);
						old[x][e] = (rr < p && cc < p) ? Q[(int64_t)cc * p + rr] : 0.0;
					}
#pragma unroll
				for (int x = 0; x < 4; x++) {
					const int r = rq + 16 * x;
					double c[4] = {0.0, 0.0, 0.0, 0.0};
					const int ra = min(r + g, p - 1), rb = min(r + g + 8, p - 1);
					const double x0[4] = {V[t * ld + ra], V[t * ld + rb], V[(t + 4) * ld + ra], V[(t + 4) * ld + rb]};
					const double x1[4] = {V[(t + 8) * ld + ra], V[(t + 8) * ld + rb], V[(t + 12) * ld + ra], V[(t + 12) * ld + rb]};
					dg_mma(c, x0, b0);
					dg_mma(c, x1, b1);
#pragma unroll
					for (int e = 0; e < 4; e++) {
						const int rr = r + g + 8 * (e >> 1), cc = c0 + 2 * t + (e & 1);
						if (rr < p && cc < p) Q[(int64_t)cc * p + rr] = old[x][e] - c[e];
					}
				}
			}
		}
	}
}

// Implicit QL iteration with Wilkinson shifts on the tridiagonal matrix, one warp per matrix (every
// lane carries the same scalars; the lanes share the search for a negligible off-diagonal entry and
// the stores of the rotations).  A rotation is a chain of about 100 cycles (one reciprocal square root),
// so the launch is bound by the order p, about 0.85 p^2 rotations, until several thousand matrices
// fill the float64 pipes.  Off-diagonal entries at or below eps ||T|| count as zero, which keeps
// the error at the level of the tridiagonalisation's own.
__global__ void __launch_bounds__(32) k_eig_ql(const EigWork *__restrict__ work, double *Sb, double *lamb, int round) {
	extern __shared__ __align__(16) double ql_sm[];
	const EigWork w = work[blockIdx.x];
	const int p = w.p, lane = threadIdx.x;
	const EigScratch L = EigScratch::make(p);
	double *S = Sb + w.s;
	EigState *st = reinterpret_cast<EigState *>(S + L.state);
	if (st->done) return;
	double *d = ql_sm, *e = ql_sm + p;
	double scale = st->scale;
	if (round == 1) {
		double mx = 0.0;
		for (int i = lane; i < p; i += 32) mx = fmax(mx, fmax(fabs(S[L.d + i]), fabs(S[L.e + i])));
		for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
		// a power of two, so that scaling is exact
		scale = (mx > 0.0 && isfinite(mx)) ? exp2((double)ilogb(mx)) : 1.0;
	}
	const double inv = round == 1 ? 1.0 / scale : 1.0;
	double tn = 0.0;
	for (int i = lane; i < p; i += 32) {
		d[i] = S[L.d + i] * inv;
		e[i] = S[L.e + i] * inv;
		tn = fmax(tn, fabs(d[i]) + fabs(e[i]));
	}
	for (int o = 16; o > 0; o >>= 1) tn = fmax(tn, __shfl_xor_sync(0xffffffffu, tn, o));
	const double thr = Eps<double>::v() * tn;
	__syncwarp();
	int2 *sweep = reinterpret_cast<int2 *>(S + L.sweep);
	double2 *rot = reinterpret_cast<double2 *>(S + L.rot);
	int ns = 0, l = st->next;
	bool full = false;
	int tries = 0;
	while (l < p) {
		// first negligible off-diagonal entry at or after l
		int m = p - 1;
		for (int b = l; b < p - 1; b += 32) {
			const bool small = b + lane < p - 1 && !(fabs(e[b + lane]) > thr);
			const unsigned bal = __ballot_sync(0xffffffffu, small);
			if (bal) {
				m = b + __ffs(bal) - 1;
				break;
			}
		}
		if (m == l) {
			l++;
			tries = 0;
			continue;
		}
		if (ns == L.cap || tries == 60) {
			full = true;
			break;
		}
		tries++;
		const double dl = d[l], el = e[l];
		double g = (d[l + 1] - dl) / (2.0 * el);
		double r = sqrt(fma(g, g, 1.0));
		g = d[m] - dl + el / (g + copysign(r, g));
		double s = 1.0, c = 1.0, q = 0.0;
		double2 mine = make_double2(1.0, 0.0);
		double dn = d[m];  // d[i + 1]
		double ei = e[m - 1], di = d[m - 1];
		// the dependent chain of a rotation: g^2, h, the reciprocal root, rr, g
		for (int i = m - 1; i >= l; i--) {
			const int ip = max(i - 1, l);
			const double en = e[ip], dp = d[ip];  // read ahead of this step's stores
			// lane 0 stores entries i + 1 below: every lane has read them (a sweep ago, or before the loop) by
			// now, whatever the pace of the lanes
			__syncwarp();
			const double f = s * ei, b = c * ei;
			const double h = fma(f, f, g * g);
			const double gg = dn - q;
			const double u = fma(di - gg, f, g * (b + b));
			const bool some = h > 0.0;  // else both vanish: nothing to rotate
			const double ri = rsqrt(h);
			s = some ? f * ri : 0.0;
			c = some ? g * ri : 1.0;
			const double rr = some ? u * ri : b + b;
			q = s * rr;
			g = fma(c, rr, -b);
			if (lane == 0) {
				e[i + 1] = some ? h * ri : 0.0;
				d[i + 1] = gg + q;
			}
			dn = di;
			di = dp;
			ei = en;
			if (lane == (i & 31)) mine = make_double2(c, s);
			if ((i & 31) == 0 || i == l) {
				const int at = (i & ~31) + lane;
				if (at >= i && at < m) rot[(int64_t)ns * p + at] = mine;
			}
		}
		__syncwarp();
		if (lane == 0) {
			d[l] = d[l] - q;
			e[l] = g;
			e[m] = 0.0;
			sweep[ns] = make_int2(l, m);
		}
		__syncwarp();
		ns++;
	}
	// eigenvalues in decreasing order (ties by index)
	int *rank = reinterpret_cast<int *>(S + L.rank);
	const bool last = !full || round == kEigRounds;
	if (last) {
		for (int i = lane; i < p; i += 32) {
			const double x = d[i];
			const double kx = isnan(x) ? INFINITY : x;  // NaN first, so that the ranks stay a permutation
			int k = 0;
			for (int o = 0; o < p; o++) {
				const double ky = isnan(d[o]) ? INFINITY : d[o];
				k += (ky > kx || (ky == kx && o < i)) ? 1 : 0;
			}
			rank[i] = k;
			lamb[w.lam + k] = x * scale;
		}
	}
	for (int i = lane; i < p; i += 32) {
		S[L.d + i] = d[i];
		S[L.e + i] = e[i];
	}
	if (lane == 0) {
		st->next = l;
		st->sweeps = ns;
		st->scale = scale;
		st->done = last ? round : 0;
		st->bad = last && full ? 1 : 0;
	}
}

// The recorded rotations applied to the rows of Q, the result written as the eigenvector columns in
// their final order (or left in Q when a further round follows).  One warp takes 32 rows, a thread
// a row, in place in Q (column-major, so a column's 32 rows are one 256-byte access).  A sweep runs
// its rotations down the columns: with x carried, column i + 1 becomes s y + c x and x becomes
// c y - s x (y = column i); rotations outside a sweep's range are the identity (c, s) = (1, 0).  Eight
// sweeps run as a pipeline, sweep k two columns behind sweep k - 1, so each element is loaded and
// stored once per eight rotations and the eight rotations of a step are independent; a rotation
// then costs its four multiply-adds.  The rows stay in L2 rather than in shared memory, where 32 of
// them would leave room for two or three warps an SM (measured 17.5 ms for 256 matrices of order
// 400); elements are read four steps ahead.
constexpr int kEigRows = 32;

__global__ void __launch_bounds__(32) k_eig_rotate(const EigWork *__restrict__ work, double *Ab, double *Qb,
                                                   const double *__restrict__ Sb, int round) {
	__shared__ __align__(16) double2 cs[2][kEigSweeps][32];
	const EigWork w = work[blockIdx.y];
	const int p = w.p, lane = threadIdx.x, r0 = blockIdx.x * kEigRows;
	if (r0 >= p) return;
	const EigScratch L = EigScratch::make(p);
	const double *S = Sb + w.s;
	const EigState st = *reinterpret_cast<const EigState *>(S + L.state);
	if (st.done && st.done < round) return;
	double *A = Ab + w.a;
	const bool own = r0 + lane < p;
	double *z = Qb + w.q + (own ? r0 + lane : p - 1);  // idle lanes read the last row and store nothing
	const int2 *sweep = reinterpret_cast<const int2 *>(S + L.sweep);
	const double2 *rot = reinterpret_cast<const double2 *>(S + L.rot);
	for (int s0 = 0; s0 < st.sweeps; s0 += kEigSweeps) {
		int lo = p, hi = 0;
		int2 rg[kEigSweeps];
#pragma unroll
		for (int k = 0; k < kEigSweeps; k++) {
			rg[k] = s0 + k < st.sweeps ? sweep[s0 + k] : make_int2(0, 0);
			if (rg[k].y > rg[k].x) {
				lo = min(lo, rg[k].x);
				hi = max(hi, rg[k].y);
			}
		}
		// step i: sweep k works on column i + 2 k with rotation i + 2 k
		const int i_end = lo - 1 - 2 * (kEigSweeps - 1);
		double2 nx[kEigSweeps];
		auto fetch = [&](int top) {  // the 32 steps top - 31 .. top: entry `lane` is step top - 31 + lane
#pragma unroll
			for (int k = 0; k < kEigSweeps; k++) {
				const int i = top - 31 + lane + 2 * k;
				nx[k] = (i >= rg[k].x && i < rg[k].y) ? rot[(int64_t)(s0 + k) * p + i] : make_double2(1.0, 0.0);
			}
		};
		auto elem = [&](int i) { return z[(int64_t)max(i, 0) * p]; };  // columns below lo meet the identity only
		double x[kEigSweeps], o[kEigSweeps], y4[4];
#pragma unroll
		for (int k = 0; k < kEigSweeps; k++) x[k] = o[k] = 0.0;
#pragma unroll
		for (int q = 0; q < 4; q++) y4[q] = elem(hi - q);
		fetch(hi);
		int buf = 0;
		for (int top = hi; top >= i_end; top -= 32, buf ^= 1) {
#pragma unroll
			for (int k = 0; k < kEigSweeps; k++) cs[buf][k][lane] = nx[k];
			__syncwarp();
			if (top - 32 >= i_end) fetch(top - 32);
			double2 r[kEigSweeps];
#pragma unroll
			for (int k = 0; k < kEigSweeps; k++) r[k] = cs[buf][k][31];
			// whole groups of four steps; those past i_end meet the identity and store nothing
			for (int i4 = 31; i4 >= 0 && top - 31 + i4 >= i_end; i4 -= 4) {
#pragma unroll
				for (int q = 0; q < 4; q++) {
					const int i = top - 31 + i4 - q;
					const double y0 = y4[q];
					y4[q] = elem(i - 4);
					double2 rn[kEigSweeps];
					const int nxt = max(i4 - q - 1, 0);
#pragma unroll
					for (int k = 0; k < kEigSweeps; k++) rn[k] = cs[buf][k][nxt];
#pragma unroll
					for (int k = kEigSweeps - 1; k >= 0; k--) {
						const double y = k ? o[k - 1] : y0;
						const double out = fma(r[k].y, y, r[k].x * x[k]);
						x[k] = fma(r[k].x, y, -r[k].y * x[k]);
						o[k] = out;
					}
					const int at = i + 2 * (kEigSweeps - 1) + 1;
					if (own && at >= lo && at <= hi) z[(int64_t)at * p] = o[kEigSweeps - 1];
#pragma unroll
					for (int k = 0; k < kEigSweeps; k++) r[k] = rn[k];
				}
			}
			__syncwarp();
		}
	}
	if (st.done != round || !own) return;
	const int *rank = reinterpret_cast<const int *>(S + L.rank);
	for (int c = 0; c < p; c++) A[(int64_t)rank[c] * p + r0 + lane] = z[(int64_t)c * p];
}

}  // namespace hab200
