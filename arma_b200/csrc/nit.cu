// Nonlinear inertialess transform (NIT) of a Gaussian surface to a target
// distribution: each value z becomes y with F_target(y) = Phi_sigma(z)
// (reference src/nonlinear/transforms.hh:58-75 driven by
// src/nonlinear/nit_transform.cc:147-168).
//
// Two forms:
//   bisection  the reference's per-point bisection (src/linalg.hh:199-213):
//              midpoint, evaluate f(c), move the bracket by the sign of
//              f(a)*f(c) and f(b)*f(c), stop after max_iter iterations or when
//              the bracket is no wider than eps or |f(c)| <= eps.  FP64, with
//              the same result and almost no evaluations (below).
//   LUT        a pointwise map through an FP64-built inverse-CDF table with
//              cubic Lagrange interpolation between nodes and linear
//              extrapolation beyond the end nodes, stored per interval as
//              power-basis coefficients (one vector load and three FMAs per
//              value).  HBM-bound: one read and one write per value.
#include <algorithm>
#include <cmath>
#include <cstdint>

#include "distributions.h"
#include "internal.h"

namespace armab {
namespace {

constexpr int kThreads = 256;

__constant__ dist::GL20 c_gl20;

// The bisection of every point walks one tree of midpoints of the interval and
// compares F(c) - target, so its first K levels read F at the tree's nodes from a
// table of 2^K + 1 values, made for the call (each node's c by the same halvings).
// Below, a level needs only the sign of F(c) - target and whether it is within
// eps: a cubic through the four nodes around the cell gives both unless it lies
// within delta of 0 or eps, and then F(c) is evaluated.  delta is eight times the
// cubic's error as estimated on the table itself (the odd nodes from the even
// ones, an error about 16 times as large), plus 90 times what F rounds to at the
// size of its terms.  Results are those of evaluating F at
// a, b and c in every iteration (25 x 3 evaluations of 11 exponentials for eps
// 1e-6 on [-10, 10]): 320000 points in 27 us instead of 815.
struct BisectTable {
	const double* f;      // F at node i = 0 .. 2^levels
	const double* error;  // largest error of the odd nodes from the even ones
	int levels;
	int cubic;            // the nodes resolve F: cubics below the table
	double inv_h;         // 1 / node distance
	double rounding;      // of F and of the cubics
};

__global__ void __launch_bounds__(kThreads)
bisect_table_kernel(double* __restrict__ f, int levels, int d, double p0, double p1, double p2,
                    double a0, double b0) {
	const int i = blockIdx.x * kThreads + threadIdx.x, n = 1 << levels;
	if (i > n) return;
	const double p[3] = {p0, p1, p2};
	double a = a0, b = b0, c = i == 0 ? a0 : b0;
	if (i > 0 && i < n) {
		int lo = 0, hi = n;
		for (;;) {
			const int mid = (lo + hi) >> 1;
			c = 0.5 * (a + b);
			if (mid == i) break;
			if (i < mid) {
				hi = mid;
				b = c;
			} else {
				lo = mid;
				a = c;
			}
		}
	}
	f[i] = dist::target_cdf(d, p, c, c_gl20);
}

// *error = the largest |odd node - cubic through the even nodes around it|; NaN
// counts as infinite
__global__ void __launch_bounds__(kThreads)
bisect_error_kernel(const double* __restrict__ f, int levels, unsigned long long* __restrict__ error) {
	const int i = 2 * (blockIdx.x * kThreads + threadIdx.x) + 3, n = 1 << levels;
	double e = 0.0;
	if (i + 3 <= n)
		e = fabs(f[i] - (0.5625 * (f[i - 1] + f[i + 1]) - 0.0625 * (f[i - 3] + f[i + 3])));
	if (!(e <= 1.0)) e = INFINITY;
	for (int o = 16; o > 0; o >>= 1) e = fmax(e, __shfl_xor_sync(0xffffffffu, e, o));
	// non-negative doubles order as their bits
	if ((threadIdx.x & 31) == 0) atomicMax(error, (unsigned long long)__double_as_longlong(e));
}

template <class T>
__global__ void __launch_bounds__(kThreads)
nit_bisection_kernel(T* __restrict__ z, unsigned long long n, int d, double p0, double p1,
                     double p2, double stdev, double a0, double b0, double eps, int max_iter,
                     const BisectTable tab) {
	const double p[3] = {p0, p1, p2};
	const dist::GL20& g = c_gl20;
	const int nodes = 1 << tab.levels;
	const double f0 = tab.f[0], f1 = tab.f[nodes];
	const double delta = tab.cubic ? 0.5 * *tab.error + tab.rounding : 0.0;
	for (unsigned long long idx = blockIdx.x * (unsigned long long)kThreads + threadIdx.x;
	     idx < n; idx += (unsigned long long)gridDim.x * kThreads) {
		const double target = dist::gaussian_cdf(double(z[idx]), 0.0, stdev);
		double a = a0, b = b0, fa = f0 - target, fb = f1 - target, c, fc;
		double x0 = 0.0, k0 = 0.0, k1 = 0.0, k2 = 0.0, k3 = 0.0;
		int lo = 0, hi = nodes, i = 0;
		bool cell = false, moved;
		do {
			c = 0.5 * (a + b);
			const int mid = (lo + hi) >> 1;
			const bool in_table = hi - lo > 1;
			if (in_table) {
				fc = tab.f[mid] - target;
			} else {
				if (!cell && tab.cubic && lo > 0 && lo + 2 <= nodes) {
					// F(x0 + t h) = k0 + k1 t + k2 t^2 + k3 t^3 through nodes
					// lo - 1 .. lo + 2 (t = -1, 0, 1, 2)
					const double m = tab.f[lo - 1], u = tab.f[lo], v = tab.f[lo + 1],
					             w = tab.f[lo + 2];
					x0 = a;
					k0 = u;
					k2 = 0.5 * (m + v) - u;
					k3 = (w - m - 3.0 * (v - u)) / 6.0;
					k1 = v - u - k2 - k3;
					cell = true;
				}
				bool evaluate = true;
				if (cell) {
					const double t = (c - x0) * tab.inv_h;
					fc = fma(fma(fma(k3, t, k2), t, k1), t, k0) - target;
					evaluate = !(fabs(fc) > delta && fabs(fabs(fc) - eps) > delta);
				}
				if (evaluate) fc = dist::target_cdf(d, p, c, g) - target;
			}
			moved = false;
			if (fa * fc < 0.0) {
				b = c;
				fb = fc;
				if (in_table) hi = mid;
				moved = true;
			}
			if (fb * fc < 0.0) {
				a = c;
				fa = fc;
				if (in_table) lo = mid;
				moved = true;
			}
			i++;
			// (a bracket that did not move stays for every later iteration)
		} while (i < max_iter && (b - a) > eps && fabs(fc) > eps && moved);
		z[idx] = T(c);
	}
}

// The table map over n values: groups of kLutPer 16-byte vectors per thread,
// all loaded before any is mapped (the loads in flight together); the ragged
// head and tail before / after the vectors scalar.  The coefficient table is
// staged in shared memory when it fits (smem = true), else read through L1.
template <class T> struct LutVec;
template <> struct LutVec<float> { using type = float4; static constexpr int n = 4; };
template <> struct LutVec<double> { using type = double2; static constexpr int n = 2; };
constexpr int kLutPer = 4;
constexpr size_t kLutSmemMax = 48 * 1024;

template <class T>
__global__ void __launch_bounds__(kThreads)
nit_lut_kernel(T* __restrict__ z, unsigned long long n,
               const typename NitCoef<T>::type* __restrict__ table, int nodes, T x0, T inv_dx,
               int smem) {
	using C = typename NitCoef<T>::type;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	const C* coef = table;
	if (smem) {
		C* s = reinterpret_cast<C*>(smem_raw);
		for (int i = threadIdx.x; i <= nodes; i += kThreads) s[i] = table[i];
		__syncthreads();
		coef = s;
	}
	using V = typename LutVec<T>::type;
	constexpr int W = LutVec<T>::n;
	// head: values before the first 16-byte boundary
	const unsigned long long head =
	    min(n, (unsigned long long)((16 - (reinterpret_cast<uintptr_t>(z) & 15)) & 15) / sizeof(T));
	const unsigned long long gtid = blockIdx.x * (unsigned long long)kThreads + threadIdx.x;
	const unsigned long long nthr = (unsigned long long)gridDim.x * kThreads;
	if (gtid < head) z[gtid] = nit_lut_map(z[gtid], coef, nodes, x0, inv_dx);
	V* zv = reinterpret_cast<V*>(z + head);
	const unsigned long long nv = (n - head) / W;
	for (unsigned long long base = gtid; base < nv; base += nthr * kLutPer) {
		V v[kLutPer];
#pragma unroll
		for (int r = 0; r < kLutPer; ++r) {
			const unsigned long long i = base + r * nthr;
			if (i < nv) v[r] = zv[i];
		}
#pragma unroll
		for (int r = 0; r < kLutPer; ++r) {
			const unsigned long long i = base + r * nthr;
			if (i < nv) {
				T* e = reinterpret_cast<T*>(&v[r]);
#pragma unroll
				for (int k = 0; k < W; ++k) e[k] = nit_lut_map(e[k], coef, nodes, x0, inv_dx);
				zv[i] = v[r];
			}
		}
	}
	for (unsigned long long i = head + nv * W + gtid; i < n; i += nthr)
		z[i] = nit_lut_map(z[i], coef, nodes, x0, inv_dx);
}

void upload_gl20(Ctx* c) {
	static bool done[64] = {false};
	if (c->device >= 0 && c->device < 64 && !done[c->device]) {
		const dist::GL20& g = dist::gl20_host();
		ARMA_CUDA_TRY(cudaMemcpyToSymbol(c_gl20, &g, sizeof(g)));
		done[c->device] = true;
	}
}

int grid_for(unsigned long long n, int sms) {
	const unsigned long long b = (n + kThreads - 1) / kThreads;
	return int(b < (unsigned long long)(sms * 8) ? (b ? b : 1) : sms * 8);
}

}  // namespace

void launch_nit_bisection(Ctx* c, int d, const double params[3], double stdev, double a,
                          double b, double eps, int max_iter, uint64_t n, int precision,
                          void* d_zeta) {
	ProfScope prof_(c, "nit");
	upload_gl20(c);
	// An iteration either moves one end of the bracket to a midpoint strictly
	// inside it, or leaves the bracket, and so every later iteration, as it
	// is.  A bracket of finite doubles can be halved at most ~2100 times
	// (2^1024 down to the subnormal spacing 2^-1074) before its midpoint
	// rounds to an end, so iterations past 4096 never change the result:
	// larger counts are cut there, which bounds the kernel's run time without
	// changing any output.
	const int iters = std::min(max_iter, 4096);
	const int grid = grid_for(n, c->num_sms);
	if (n == 0) return;
	// table levels: up to 2^16 nodes, at most a quarter of the points
	BisectTable tab{};
	const bool proper = std::isfinite(a) && std::isfinite(b) && a < b;
	while (proper && tab.levels < 16 && (8ull << tab.levels) <= n) ++tab.levels;
	const int nodes = 1 << tab.levels;
	const double h = (b - a) / nodes;
	// cubics where the nodes resolve the distribution: its finest features are
	// those of width stdev / sqrt(1 + alpha^2) of the skew normal's T, or about 1
	const double width = d == ARMA_NIT_SKEW_NORMAL
	                         ? std::fabs(params[1]) / std::sqrt(1.0 + params[2] * params[2])
	                         : 1.0;
	tab.cubic = proper && tab.levels >= 6 && h <= 0.05 * width;
	tab.inv_h = 1.0 / h;
	// F's terms: |x|^k exp(-x^2 / 2) is at most 0.61, 0.74, 1.16 for k = 1, 2, 3 (and
	// 1 / (24 sqrt(2 pi)) 0.0167); Owen's T sums up to |alpha|
	const double s = std::fabs(params[0]), k = std::fabs(params[1]);
	const double terms = d == ARMA_NIT_SKEW_NORMAL
	                         ? 1.0 + std::fabs(params[2])
	                         : 1.0 + 0.0167 * ((3 * 0.61 + 1.16) * k + (4 + 4 * 0.74) * s + 9.0);
	tab.rounding = 1e-14 * terms;
	auto* f = static_cast<double*>(scratch_take(c, sizeof(double) * (size_t(nodes) + 1)));
	auto* error = static_cast<unsigned long long*>(scratch_take(c, sizeof(double)));
	tab.f = f;
	tab.error = reinterpret_cast<const double*>(error);
	bisect_table_kernel<<<nodes / kThreads + 1, kThreads, 0, c->stream>>>(
	    f, tab.levels, d, params[0], params[1], params[2], a, b);
	ARMA_CUDA_TRY(cudaGetLastError());
	c->launches += 1;
	if (tab.cubic) {
		ARMA_CUDA_TRY(cudaMemsetAsync(error, 0, sizeof(double), c->stream));
		bisect_error_kernel<<<nodes / 2 / kThreads + 1, kThreads, 0, c->stream>>>(f, tab.levels,
		                                                                          error);
		ARMA_CUDA_TRY(cudaGetLastError());
		c->launches += 1;
	}
	if (precision == ARMA_FP64)
		nit_bisection_kernel<double><<<grid, kThreads, 0, c->stream>>>(
		    static_cast<double*>(d_zeta), n, d, params[0], params[1], params[2], stdev, a, b,
		    eps, iters, tab);
	else
		nit_bisection_kernel<float><<<grid, kThreads, 0, c->stream>>>(
		    static_cast<float*>(d_zeta), n, d, params[0], params[1], params[2], stdev, a, b,
		    eps, iters, tab);
	ARMA_CUDA_TRY(cudaGetLastError());
	c->launches += 1;
}

void launch_nit_lut(Ctx* c, const void* d_coef, int nodes, double x0, double dx,
                    uint64_t n, int precision, void* d_zeta) {
	ProfScope prof_(c, "nit");
	ARMA_REQUIRE(nodes >= 4, ARMA_EINVAL, "NIT table needs at least 4 nodes");
	const int grid = grid_for(n, c->num_sms);
	if (precision == ARMA_FP64) {
		const size_t bytes = sizeof(double4) * (size_t(nodes) + 1);
		const bool smem = bytes <= kLutSmemMax;
		nit_lut_kernel<double><<<grid, kThreads, smem ? bytes : 0, c->stream>>>(
		    static_cast<double*>(d_zeta), n, static_cast<const double4*>(d_coef), nodes, x0,
		    1.0 / dx, smem);
	} else {
		const size_t bytes = sizeof(float4) * (size_t(nodes) + 1);
		const bool smem = bytes <= kLutSmemMax;
		nit_lut_kernel<float><<<grid, kThreads, smem ? bytes : 0, c->stream>>>(
		    static_cast<float*>(d_zeta), n, static_cast<const float4*>(d_coef), nodes,
		    float(x0), float(1.0 / dx), smem);
	}
	ARMA_CUDA_TRY(cudaGetLastError());
	c->launches += 1;
}

}  // namespace armab
