// Circular auto-covariance of a 3-D array on the device: the reference's
// arma::auto_covariance (src/arma.cc:81-100), Re IFFT(|FFT(w)|^2) / n / n,
// which its wave-group ACF generator (src/generator/acf_generator.cc:147) and
// its ACF checks of generated surfaces use.
//
// FP64 throughout, sides up to kMaxLine (the ACF generator works on 2 nwaves + 1
// <= 129 points per axis, a realisation's ACF check on its own sides).  The input
// is real, so only ny / 2 + 1 of the last axis's frequencies are kept; five
// passes over that half spectrum, each transforming a band of lines in shared
// memory:
//   rows    two lines of y packed as one complex line, forward, unpacked
//   x       forward, left in digit-reversed order (nothing needs its order)
//   t       forward, |.|^2, inverse
//   x       inverse
//   rows    two lines packed, inverse, / n / n
// Mixed-radix lines (fft_band): butterflies of 2, 3, 4, 5 and 7 in place, any
// other prime by direct summation, one output per thread.
//
// Bound by the lines' butterflies (their index arithmetic and shared-memory
// round trips; the passes move 0.5 GB, 80 us): 256 x 128 x 128 FP64 167 us; one
// complex pass per axis with every line by direct summation took 5540 us.  Bands
// of 3072 points: 1024 ran 20 to 40 % slower, 4096 the same.
#include <algorithm>
#include <cmath>

#include "internal.h"

namespace armab {
namespace {

constexpr int kAcThreads = 256;
constexpr int kMaxLine = 1024;
constexpr int kAcStages = 10;          // 2^10 = 1024
constexpr int kAcBand = 3072;          // most points of a band (48 KB)
constexpr int kAcLeast = 256;          // fewest

struct AcPlan {
	int n, m;
	int r[kAcStages];
	int h[kAcStages], tws[kAcStages];  // sub-block length, twiddle stride n / (r h)
	Divider by_h[kAcStages], by_per[kAcStages], by_r[kAcStages];  // per: work items of a line
	bool spare;  // a direct stage: the band needs a second buffer
};

AcPlan ac_plan(int n) {
	AcPlan p{};
	p.n = n;
	int rest = n;
	for (int f : {4, 2, 3, 5, 7})
		while (rest % f == 0) {
			p.r[p.m++] = f;
			rest /= f;
		}
	for (int f = 11; rest > 1; f += 2)
		while (rest % f == 0) {
			p.r[p.m++] = f;
			rest /= f;
			p.spare = true;
		}
	int L = n;
	for (int s = 0; s < p.m; ++s) {
		const int r = p.r[s];
		p.h[s] = L / r;
		p.tws[s] = n / L;
		p.by_h[s] = Divider(p.h[s]);
		p.by_per[s] = Divider(r > 7 ? n : n / r);
		p.by_r[s] = Divider(r);
		L = p.h[s];
	}
	return p;
}

__device__ __forceinline__ double2 operator+(double2 a, double2 b) {
	return make_double2(a.x + b.x, a.y + b.y);
}
__device__ __forceinline__ double2 operator-(double2 a, double2 b) {
	return make_double2(a.x - b.x, a.y - b.y);
}
// a w, or a conj(w) for the inverse
template <bool INV>
__device__ __forceinline__ double2 mul_root(double2 a, double2 w) {
	const double s = INV ? -w.y : w.y;
	return make_double2(fma(a.x, w.x, -a.y * s), fma(a.x, s, a.y * w.x));
}
template <bool INV>
__device__ __forceinline__ double2 mul_minus_i(double2 a) {
	return INV ? make_double2(-a.y, a.x) : make_double2(a.y, -a.x);
}

// roots[k] = exp(-2 pi i k / n) of the three axes, one after another
__global__ void roots_kernel(double2* __restrict__ roots, int n0, int n1, int n2) {
	const int q = blockIdx.x * kAcThreads + threadIdx.x;
	if (q >= n0 + n1 + n2) return;
	const int n = q < n0 ? n0 : q < n0 + n1 ? n1 : n2;
	const int k = q < n0 ? q : q < n0 + n1 ? q - n0 : q - n0 - n1;
	double s, c;
	sincospi(2.0 * k / n, &s, &c);
	roots[q] = make_double2(c, -s);
}

__device__ void ac_twiddles(double2* tw, const double2* __restrict__ roots, int n) {
	for (int k = threadIdx.x; k < n; k += kAcThreads) tw[k] = roots[k];
}

template <bool INV, int R>
__device__ __forceinline__ void ac_butterfly(double2* x, int hs, int step, int rs, const double2* tw) {
	double2 v[R];
#pragma unroll
	for (int k = 0; k < R; ++k) v[k] = x[k * hs];
	if (INV) {
#pragma unroll
		for (int k = 1; k < R; ++k) v[k] = mul_root<true>(v[k], tw[k * step]);
	}
	if constexpr (R == 2) {
		const double2 a = v[0];
		v[0] = a + v[1];
		v[1] = a - v[1];
	} else if constexpr (R == 4) {
		const double2 t0 = v[0] + v[2], t1 = v[0] - v[2], t2 = v[1] + v[3];
		const double2 t3 = mul_minus_i<INV>(v[1] - v[3]);
		v[0] = t0 + t2;
		v[1] = t1 + t3;
		v[2] = t0 - t2;
		v[3] = t1 - t3;
	} else {
		double2 y[R];
#pragma unroll
		for (int q = 0; q < R; ++q) {
			y[q] = v[0];
#pragma unroll
			for (int k = 1; k < R; ++k) y[q] = y[q] + mul_root<INV>(v[k], tw[(q * k) % R * rs]);
		}
#pragma unroll
		for (int q = 0; q < R; ++q) v[q] = y[q];
	}
	if (!INV) {
#pragma unroll
		for (int k = 1; k < R; ++k) v[k] = mul_root<false>(v[k], tw[k * step]);
	}
#pragma unroll
	for (int k = 0; k < R; ++k) x[k * hs] = v[k];
}

// (out of line: their registers would halve the warps on an SM)
template <bool INV, int R>
__device__ __noinline__ void ac_butterfly_call(double2* x, int hs, int step, int rs,
                                               const double2* tw) {
	ac_butterfly<INV, R>(x, hs, step, rs, tw);
}

// FFTs of `lines` lines (line l, element e at l ls + e es of the band; lines *
// n < 2^16) in buffer a, b a second one where the plan needs it; returns the
// buffer that holds the result.  Forward: decimation in frequency, position sum
// q_s h_s of the output holds frequency sum q_s r_0 .. r_(s-1); the inverse
// mirrors it.  Unnormalised.  across: neighbouring threads take neighbouring
// lines (column bands), else neighbouring elements.
template <bool INV>
__device__ double2* fft_band(double2* a, double2* b, int lines, int ls, int es, const AcPlan& P,
                             const double2* tw, bool across) {
	const int n = P.n;
	const Divider by_lines(lines);
	for (int si = 0; si < P.m; ++si) {
		const int st = INV ? P.m - 1 - si : si;
		const int r = P.r[st], h = P.h[st], L = r * h, tws = P.tws[st], rs = tws * h;
		const bool direct = r > 7;
		const int per = int(P.by_per[st].d);
		const bool by_line = across || (h < 32 && lines >= 8);
		const Divider dl = by_line ? by_lines : P.by_per[st], dh = P.by_h[st], dr = P.by_r[st];
		for (int q = threadIdx.x; q < lines * per; q += kAcThreads) {
			const int hi = dl.div(q), lo = q - hi * int(dl.d);
			const int line = by_line ? lo : hi, w = by_line ? hi : lo;
			int blk = dh.div(w);
			const int j = w - blk * h;
			if (!direct) {
				double2* x = a + line * ls + (blk * L + j) * es;
				switch (r) {
					case 4: ac_butterfly<INV, 4>(x, h * es, j * tws, rs, tw); break;
					case 2: ac_butterfly<INV, 2>(x, h * es, j * tws, rs, tw); break;
					case 3: ac_butterfly<INV, 3>(x, h * es, j * tws, rs, tw); break;
					case 5: ac_butterfly_call<INV, 5>(x, h * es, j * tws, rs, tw); break;
					default: ac_butterfly_call<INV, 7>(x, h * es, j * tws, rs, tw); break;
				}
			} else {
				// output p of the block: sum_k x_k W_L^(k p h) W_L^(p j), or its
				// mirror sum_k x_k conj W_L^(k (j + p h))
				const int b0 = dr.div(blk), p = blk - b0 * r;
				const double2* x = a + line * ls + (b0 * L + j) * es;
				const int step = (INV ? j + p * h : p * h) * tws;  // < n
				double2 acc = make_double2(0.0, 0.0);
				int k = 0;
				for (int i = 0; i < r; ++i) {
					acc = acc + mul_root<INV>(x[i * h * es], tw[k]);
					k += step;
					if (k >= n) k -= n;
				}
				if (!INV) acc = mul_root<false>(acc, tw[p * j * tws]);
				b[line * ls + (b0 * L + j + p * h) * es] = acc;
			}
		}
		__syncthreads();
		if (direct) {
			double2* t = a;
			a = b;
			b = t;
		}
	}
	return a;
}

// Where the forward transform leaves each frequency.
__device__ void ac_positions(int* pos, const AcPlan& P) {
	for (int p = threadIdx.x; p < P.n; p += kAcThreads) {
		int rest = p, w = 1, f = 0;
		for (int s = 0; s < P.m; ++s) {
			const int q = P.by_h[s].div(rest);
			f += q * w;
			rest -= q * P.h[s];
			w *= P.r[s];
		}
		pos[f] = p;
	}
}

// Shared memory of a band: points, a second buffer where the plan needs it, n
// twiddles, n positions.
size_t ac_smem(const AcPlan& P, int points) {
	return sizeof(double2) * (size_t(points) * (P.spare ? 2 : 1) + P.n) + sizeof(int) * size_t(P.n);
}

struct Band {
	double2 *a, *b, *tw;
	int* pos;
	__device__ Band(double2* smem, const AcPlan& P, int points)
	    : a(smem), b(P.spare ? smem + points : smem), tw(b + points), pos(reinterpret_cast<int*>(tw + P.n)) {}
};

// Two real lines of n values as the real and imaginary part of one complex line:
// lines 2 q and 2 q + 1 of the array, `pairs` of them per CTA, into the half
// spectrum w (line l, frequency k at l nh + k).
template <class T>
__global__ void __launch_bounds__(kAcThreads, 3)
rows_forward_kernel(const T* __restrict__ in, double2* __restrict__ w, long long lines, int pairs,
                    const double2* __restrict__ roots, const AcPlan P) {
	extern __shared__ __align__(16) double2 ac_mem[];
	const int n = P.n, ld = n + 1, nh = n / 2 + 1;
	const Band s(ac_mem, P, pairs * ld);
	const long long l0 = 2ll * blockIdx.x * pairs;
	const int here = int(min((long long)pairs, (lines - l0 + 1) / 2));
	ac_twiddles(s.tw, roots, n);
	ac_positions(s.pos, P);
	for (int q = threadIdx.x; q < here * n; q += kAcThreads) {
		const int i = q / n, e = q - i * n;
		const long long l = l0 + 2 * i;
		s.a[i * ld + e] = make_double2(double(in[l * n + e]),
		                               l + 1 < lines ? double(in[(l + 1) * n + e]) : 0.0);
	}
	__syncthreads();
	const double2* z = fft_band<false>(s.a, s.b, here, ld, 1, P, s.tw, false);
	for (int q = threadIdx.x; q < here * nh; q += kAcThreads) {
		const int i = q / nh, k = q - i * nh;
		const long long l = l0 + 2 * i;
		const double2 u = z[i * ld + s.pos[k]], v = z[i * ld + s.pos[k == 0 ? 0 : n - k]];
		w[l * nh + k] = make_double2(0.5 * (u.x + v.x), 0.5 * (u.y - v.y));
		if (l + 1 < lines) w[(l + 1) * nh + k] = make_double2(0.5 * (u.y + v.y), 0.5 * (v.x - u.x));
	}
}

__global__ void __launch_bounds__(kAcThreads, 3)
rows_inverse_kernel(const double2* __restrict__ w, double* __restrict__ out, long long lines,
                    int pairs, double nn, const double2* __restrict__ roots, const AcPlan P) {
	extern __shared__ __align__(16) double2 ac_mem[];
	const int n = P.n, ld = n + 1, nh = n / 2 + 1;
	const Band s(ac_mem, P, pairs * ld);
	const long long l0 = 2ll * blockIdx.x * pairs;
	const int here = int(min((long long)pairs, (lines - l0 + 1) / 2));
	ac_twiddles(s.tw, roots, n);
	ac_positions(s.pos, P);
	__syncthreads();
	for (int q = threadIdx.x; q < here * nh; q += kAcThreads) {
		const int i = q / nh, k = q - i * nh;
		const long long l = l0 + 2 * i;
		const double2 u = w[l * nh + k];
		const double2 v = l + 1 < lines ? w[(l + 1) * nh + k] : make_double2(0.0, 0.0);
		s.a[i * ld + s.pos[k]] = make_double2(u.x - v.y, u.y + v.x);
		if (k > 0 && 2 * k != n) s.a[i * ld + s.pos[n - k]] = make_double2(u.x + v.y, v.x - u.y);
	}
	__syncthreads();
	const double2* z = fft_band<true>(s.a, s.b, here, ld, 1, P, s.tw, false);
	for (int q = threadIdx.x; q < here * n; q += kAcThreads) {
		const int i = q / n, e = q - i * n;
		const long long l = l0 + 2 * i;
		const double2 v = z[i * ld + e];
		out[l * n + e] = v.x / nn / nn;
		if (l + 1 < lines) out[(l + 1) * n + e] = v.y / nn / nn;
	}
}

// Columns: element e of column c of slab blockIdx.y at slab n cols + e cols + c;
// `band` columns per CTA.  What: 0 forward, 1 inverse, 2 forward, |.|^2, inverse.
template <int WHAT>
__global__ void __launch_bounds__(kAcThreads, 3)
columns_kernel(double2* __restrict__ w, int cols, int band, const double2* __restrict__ roots,
               const AcPlan P) {
	extern __shared__ __align__(16) double2 ac_mem[];
	const int n = P.n;
	const Band s(ac_mem, P, n * band);
	const int c0 = blockIdx.x * band, here = min(band, cols - c0);
	double2* base = w + (long long)blockIdx.y * n * cols + c0;
	ac_twiddles(s.tw, roots, n);
	const Divider dc(here);
	for (int q = threadIdx.x; q < n * here; q += kAcThreads) {
		const int e = dc.div(q);
		s.a[q] = base[(long long)e * cols + q - e * here];
	}
	__syncthreads();
	double2 *z = s.a, *spare = s.b;
	if (WHAT != 1) {
		z = fft_band<false>(z, spare, here, 1, here, P, s.tw, true);
		spare = z == s.a ? s.b : s.a;
	}
	if (WHAT == 2) {
		for (int q = threadIdx.x; q < n * here; q += kAcThreads)
			z[q] = make_double2(z[q].x * z[q].x + z[q].y * z[q].y, 0.0);
		__syncthreads();
	}
	if (WHAT != 0) z = fft_band<true>(z, spare, here, 1, here, P, s.tw, true);
	for (int q = threadIdx.x; q < n * here; q += kAcThreads) {
		const int e = dc.div(q);
		base[(long long)e * cols + q - e * here] = z[q];
	}
}

// Points of a band: enough bands for four per SM, within [kAcLeast, kAcBand].
int band_points(Ctx* c, long long total) {
	return int(std::min<long long>(kAcBand, std::max<long long>(kAcLeast, total / (4ll * c->num_sms))));
}

// Columns per CTA: about `points` points, at least four (64 bytes of a row) where
// those make a CTA per SM, fewer down to one where not (lines of a large prime are
// long and few: 1021 x 2 x 2 976 -> 411 us); the bands of a row equally wide.
int columns_per_band(Ctx* c, long long slabs, int n, int cols, int points) {
	const int least = int(std::min(4ll, std::max(1ll, slabs * cols / c->num_sms)));
	const int most = std::max(least, points / n);
	const int bands = (cols + most - 1) / most;
	return (cols + bands - 1) / bands;
}

template <int WHAT>
void launch_columns(Ctx* c, double2* w, long long slabs, int cols, const double2* roots,
                    const AcPlan& P) {
	const int band = columns_per_band(c, slabs, P.n, cols, band_points(c, slabs * P.n * cols));
	const size_t smem = ac_smem(P, P.n * band);
	allow_smem(columns_kernel<WHAT>, smem);
	columns_kernel<WHAT><<<dim3((cols + band - 1) / band, unsigned(slabs)), kAcThreads, smem,
	                       c->stream>>>(w, cols, band, roots, P);
	ARMA_CUDA_TRY(cudaGetLastError());
	c->launches += 1;
}

}  // namespace

void launch_auto_covariance(Ctx* c, const void* d_in, const int shape[3], int precision,
                            double* d_out) {
	ProfScope prof_(c, "autocov");
	for (int a = 0; a < 3; ++a)
		ARMA_REQUIRE(shape[a] >= 1 && shape[a] <= kMaxLine, ARMA_ENOTSUP,
		             "auto-covariance: sides must be in [1, 1024]");
	const int nt = shape[0], nx = shape[1], ny = shape[2], nh = ny / 2 + 1;
	const long long lines = (long long)nt * nx;
	const AcPlan pt = ac_plan(nt), px = ac_plan(nx), py = ac_plan(ny);
	auto* w = static_cast<double2*>(scratch_take(c, sizeof(double2) * size_t(lines) * nh));
	auto* roots = static_cast<double2*>(scratch_take(c, sizeof(double2) * size_t(nt + nx + ny)));
	const double2 *rt = roots, *rx = roots + nt, *ry = roots + nt + nx;
	roots_kernel<<<(nt + nx + ny + kAcThreads - 1) / kAcThreads, kAcThreads, 0, c->stream>>>(
	    roots, nt, nx, ny);
	const int pairs = int(std::min<long long>((lines + 1) / 2, std::max(1, band_points(c, lines / 2 * ny) / (ny + 1))));
	const size_t smem = ac_smem(py, pairs * (ny + 1));
	const unsigned grid = unsigned(((lines + 1) / 2 + pairs - 1) / pairs);
	if (precision == ARMA_FP64) {
		allow_smem(rows_forward_kernel<double>, smem);
		rows_forward_kernel<double><<<grid, kAcThreads, smem, c->stream>>>(
		    static_cast<const double*>(d_in), w, lines, pairs, ry, py);
	} else {
		allow_smem(rows_forward_kernel<float>, smem);
		rows_forward_kernel<float><<<grid, kAcThreads, smem, c->stream>>>(
		    static_cast<const float*>(d_in), w, lines, pairs, ry, py);
	}
	ARMA_CUDA_TRY(cudaGetLastError());
	if (nx > 1) launch_columns<0>(c, w, nt, nh, rx, px);
	launch_columns<2>(c, w, 1, nx * nh, rt, pt);
	if (nx > 1) launch_columns<1>(c, w, nt, nh, rx, px);
	allow_smem(rows_inverse_kernel, smem);
	rows_inverse_kernel<<<grid, kAcThreads, smem, c->stream>>>(
	    w, d_out, lines, pairs, double((long long)nt * nx * ny), ry, py);
	ARMA_CUDA_TRY(cudaGetLastError());
	c->launches += 3;
}

}  // namespace armab
