// Plain FP64 AR filter with the reference's exact summation order.
//
// ar_generate_surface (reference src/generator/ar_model_surf.cc:5-36) updates
// zeta in place in C order; each point sums phi(k,i,j) * zeta(t-k,x-i,y-j)
// over k, i, j ascending (truncated at the array start) into a running sum
// that starts at 0, then adds the sum to the noise already stored at the
// point.  The sum is one chain of P explicitly rounded multiplies and adds (no
// FMA contraction), so the result is bit-identical to the CPU.
//
// What bounds it.  A point's chain starts with its newest neighbour, (t,x,y-1),
// so points run in parallel only on a hyperplane t+x+y = s, and a surface takes
// nt+nx+ny-2 steps of P dependent additions, 8 cycles each: 2.7 ms for 400 x 128
// x 128 of order 10^3 at 1965 MHz, whose arithmetic alone (a multiply and an add
// per tap, 64 lanes of either per cycle and SM) takes 0.70 ms.
//
// One persistent launch covers any number of surfaces.  With u = x + y the
// points of step s are t = s - u: a CTA owns a tile of TX rows x TU values of u
// (a parallelogram in x, y) and walks the steps, a compute thread per cell.
// Shared memory holds the last slices of the tile and its halo, by time (slot t
// mod depth), zero outside the surface: a zero operand adds +-0, which leaves a
// sum that starts at +0 as it is, so the chains need no truncation (coefficients
// must be finite for that: others take the hyperplane kernel at the end of this
// file).  A row of taps is read from there two rows ahead of its additions.  A
// tile's halo comes from tiles with smaller x or u; a halo warp polls their step
// counters and copies the new values from global memory, up to kMaxAhead steps
// before their use, and a publication warp releases the tile's own counter, both
// off the compute warps' path.  Tickets are handed out in dependency order, so a
// CTA only waits on tiles that running CTAs own; every wait is bounded.
//
// Measured (B200, the filter alone): 400 x 128 x 128 of order 10^3 4.9 ms (one
// launch per hyperplane, its taps read through L1: 70 ms); 200 x 40 x 40 of order
// 7^3 0.66 ms.  The step is bound by shared memory: a warp's operand takes two
// cycles of it and a broadcast pair of taps two more, so a step's tap takes 24
// cycles with eight warps of one cell per thread on an SM, 14 with four, 11 with
// two, against 8.2 for the chain.  Where throughput counts, a thread owns two
// cells, (x, y) and (x+1, y-1) of one u, that share the taps and all but one
// operand of a row (compute_pairs): four warps then move 256 cells in 21 cycles, 16
// mixed surfaces 11.9 -> 10.2 ms (9.4 by anti-diagonals, launch_tiles).  Two warps of pairs are no faster than four of
// single cells (13.5 and 13.9): a lone warp's issue bounds them.
#include <algorithm>
#include <climits>
#include <cmath>
#include <utility>
#include <vector>

#include "internal.h"

namespace armab {
namespace {

constexpr int kSpinLimit = 1 << 24;
constexpr size_t kSmemLimit = 227 * 1024 - 64;  // less the kernel's static shared memory
constexpr int kMaxAhead = 4;   // steps of halo kept ahead of their use
constexpr int kUpstream = 5;   // tiles a tile's halo can come from
constexpr int kBatch = 8;      // halo loads in flight per lane
constexpr int kLead = 2;       // doubles before the ring: pairs load one column past its left edge
constexpr int kPairTaps = 10;  // taps per row up to which two cells' operands fit in registers

struct Task64 {
	int nt, nx, ny, pt, px, py;
	int nbx, nc;      // tile rows, tiles per tile row
	int ticket_base;
	int ahead;        // halo steps kept ahead of their use
	double* zeta;
	const double* phi;
	int* flags;       // per tile: the step (t + u) up to which it is done
	const int* tiles; // tile of each ticket, or null: row by row
};

// Layout of a tile's shared memory (doubles unless said otherwise).
struct Layout64 {
	int ld, slot, depth, phi, entries;
	size_t bytes;
};

__host__ __device__ inline int even_up(int n) { return (n + 1) & ~1; }

// Ring rows: TX plus px-1 above; columns: TU plus px+py-2 to the left.  A slot
// is a multiple of 16 doubles, so that lanes of consecutive u (consecutive
// columns of consecutive slots) fall in different banks.
__host__ __device__ inline Layout64 layout64(int tx, int tu, int pt, int px, int py, int ahead) {
	Layout64 l;
	l.ld = tu + px + py - 2;
	l.slot = ((tx + px - 1) * l.ld + 15) & ~15;
	l.depth = tu + pt - 1 + ahead;
	l.phi = (pt * px + 2) * even_up(py);  // and two rows that are loaded past the last
	l.entries = (px - 1) * (tu + px + py - 2) + tx * (px + py - 2);
	l.bytes = sizeof(double) * (kLead + size_t(l.slot) * l.depth + l.phi + even_up(l.entries));
	return l;
}

__device__ __forceinline__ int ld_acquire_gpu(const int* p) {
	int v;
	asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
	return v;
}
__device__ __forceinline__ void st_release_gpu(int* p, int v) {
	asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ int ld_acquire_cta(const int* p) {
	int v;
	const unsigned a = static_cast<unsigned>(__cvta_generic_to_shared(p));
	asm volatile("ld.acquire.cta.shared.b32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
	return v;
}
__device__ __forceinline__ void st_release_cta(int* p, int v) {
	const unsigned a = static_cast<unsigned>(__cvta_generic_to_shared(p));
	asm volatile("st.release.cta.shared.b32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ void bar_sync(int id, int n) {
	asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int n) {
	asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory");
}

// Shared memory by 32-bit address (bytes), in program order: the loads stay
// where they are written, ahead of their use and spread among the arithmetic.
__device__ __forceinline__ double lds64(unsigned a) {
	double v;
	asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a));
	return v;
}
__device__ __forceinline__ void lds128(unsigned a, double& u, double& v) {
	asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(u), "=d"(v) : "r"(a));
}

// (volatile: not moved into the next row's block)
__device__ __forceinline__ double mul_here(double a, double b) {
	double v;
	asm volatile("mul.rn.f64 %0, %1, %2;" : "=d"(v) : "d"(a), "d"(b));
	return v;
}

// One row of taps in three stages at once: the products m of this row are added
// to the chain; the next row's products (taps c times window w) take their
// place; the window (at zn) and taps (at cn) of the row after that load into w
// and c as those are used up.  No addition waits for a product or a load of its
// own row, so the chain runs at the add's latency.
template <int PY, int M>
__device__ __forceinline__ void row_step(double& s, double (&m)[PY], double (&w)[PY],
                                         double (&c)[M], unsigned zn, unsigned cn) {
#pragma unroll
	for (int j = 0; j < PY; ++j) {
		s = __dadd_rn(s, m[j]);
		m[j] = mul_here(c[j], w[j]);
		w[j] = lds64(zn - 8 * j);
		if (j % 2 == 1 || j == PY - 1) lds128(cn + 8 * (j & ~1), c[j & ~1], c[(j & ~1) + 1]);
	}
}

__device__ __forceinline__ void lds64_if(double& v, unsigned a, int on) {
	asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %2, 0;\n\t"
	             "@q ld.shared.f64 %0, [%1];\n\t}" : "+d"(v) : "r"(a), "r"(on));
}

// The same for two cells: the products m0, m1 of this row are added to the two
// chains; the next row's products take their place, its taps pc times its window
// wc (chain 0) and the window before that, wp, one column on (chain 1); the window
// (at zn) and taps (at pn_a) of the row after that load into wp, as that is used
// up, and pn.  start: the row after next starts a slice, whose first window of
// chain 1 (at zs) replaces wc as that is used up; by predicate, since a branch per
// row costs a lone warp about 30 cycles of a row's 80.
template <int PY, int N, int M>
__device__ __forceinline__ void pair_step(double& s0, double& s1, double (&m0)[PY],
                                         double (&m1)[PY], double (&wc)[N], double (&wp)[N],
                                         const double (&pc)[M], double (&pn)[M], unsigned zn,
                                         unsigned pn_a, unsigned zs, int start) {
#pragma unroll
	for (int j = 0; j < PY; ++j) {
		if (j % 2 == 0) lds128(pn_a + 8 * j, pn[j], pn[j + 1]);
		s0 = __dadd_rn(s0, m0[j]);
		s1 = __dadd_rn(s1, m1[j]);
		m0[j] = mul_here(pc[j], wc[j]);
		m1[j] = mul_here(pc[j], wp[j + 1]);
		wp[j] = lds64(zn - 8 * j);
		if (j > 0) lds64_if(wc[j], zs - 8 * j, start);
	}
	wp[PY] = lds64(zn - 8 * PY);
	lds64_if(wc[PY], zs - 8 * PY, start);
}

// What the warps of a CTA share about the current tile, and its named barriers
// (0 is __syncthreads).  Step n of the compute warps ends at kBarHalo + n %
// kHaloBars, where the halo warp has arrived when it has brought in step n + 1's
// halo (up to kMaxAhead steps early), and each step's global stores are handed
// over at kBarPub + n % kPubBars, which the compute warps only arrive at (up to
// kPubBars steps early).
struct Shared64 {
	int done;       // steps completed by the compute warps
	int published;  // steps whose stores the publication warp has taken over
};
constexpr int kHaloBars = kMaxAhead + 1, kPubBars = 8;
constexpr int kBarHalo = 1, kBarPub = kBarHalo + kHaloBars;
static_assert(kBarPub + kPubBars <= 16, "named barriers");

// The halo warp: a list of the halo's cells inside the surface (offset in a slice, which
// has less than 2^31 points; place in a ring slot and lag in steps), then step
// after step their new values.  A cell in row x' and column u' = U0 + d is read
// from column max(U0, u' + b) of the tile on (b = X0 - x' rows above it, 0
// beside it), so step n of the tile brings in its value of t = n - max(0, d +
// b): a value that its owner computed at least max(1, b) steps before.  Tiles
// further up than the five polled here are therefore covered by those, whose
// own steps waited for them.  A wait that runs out sets the error word and lets
// the compute warps run on without the halo: they end, and the call fails.
template <int TX, int TU, int NC, int POLLS>
__device__ __forceinline__ void halo_warp(const Task64& tk, int bx, int c, const Layout64& L, double* ring,
                          int2* cells, Shared64* sh, int* err) {
	const int lane = threadIdx.x & 31;
	const int px = tk.px, left = px + tk.py - 2;
	const int X0 = bx * TX, U0 = X0 + c * TU;
	const int steps = tk.nt + TU - 1;
	const int top = (px - 1) * (TU + left), all = top + TX * left;
	int count = 0;
	for (int q0 = 0; q0 < all; q0 += 32) {
		const int q = q0 + lane;
		int row = 0, col = 0;
		if (q < top) {
			row = q / (TU + left);
			col = q % (TU + left);
		} else if (q < all) {
			row = px - 1 + (q - top) / left;
			col = (q - top) % left;
		}
		const int x = X0 + row - (px - 1), d = col - left, y = U0 + d - x;
		const int rel = max(0, d + max(0, X0 - x));
		const bool ok = q < all && rel < TU && x >= 0 && x < tk.nx && y >= 0 && y < tk.ny;
		const unsigned m = __ballot_sync(0xffffffffu, ok);
		if (ok)
			cells[count + __popc(m & ((1u << lane) - 1))] =
			    make_int2(x * tk.ny + y, (row * L.ld + col) << 8 | rel);
		count += __popc(m);
	}
	__syncwarp();
	// the tiles they come from: two to the left, three above
	const int* flag = nullptr;
	int known = INT_MAX;  // the owner's steps t + u' below this are done
	if (lane < kUpstream) {
		const int ub = lane < 2 ? bx : bx - 1;
		const int uc = lane < 2 ? c - 1 - lane : c + 1 - (lane - 2);
		if (ub >= 0 && uc >= 0 && uc < tk.nc) {
			flag = tk.flags + ub * tk.nc + uc;
			known = ub * TX + uc * TU;
		}
	}
	constexpr int kThreads = NC + 32;
	const long long plane = (long long)tk.nx * tk.ny;
	int n = 0;
	bool failed = false;
	while (n < steps) {
		// the steps n .. hi whose upstream values are there and whose ring
		// slots are free (and whose barriers' previous round is over)
		int hi = -1;
		for (int it = 0; it < POLLS; ++it) {
			const int freed = ld_acquire_cta(&sh->done) + tk.ahead;
			hi = min(freed, known == INT_MAX ? INT_MAX : known - U0);
			hi = min(__reduce_min_sync(0xffffffffu, hi), steps - 1);
			if (hi >= n) break;
			if (flag) known = max(known, ld_acquire_gpu(flag));
			if ((it & 63) == 63 && *((volatile int*)err) != DEV_OK) failed = true;
			if (__any_sync(0xffffffffu, failed)) break;
			if (it > 0) __nanosleep(20);
		}
		if (hi < n) {  // no more waiting for the tiles upstream
			if (lane == 0) atomicCAS(err, DEV_OK, DEV_TIMEOUT);
			flag = nullptr;
			known = INT_MAX;
			failed = false;
			continue;
		}
		// every (step, cell) of them, kBatch loads in flight per lane
		const int total = (hi - n + 1) * count;
		int e = lane, st = n, sm = n % L.depth;
		auto settle = [&] {
			while (e >= count) {
				e -= count;
				++st;
				sm = sm + 1 == L.depth ? 0 : sm + 1;
			}
		};
		for (int q0 = lane; q0 < total; q0 += 32 * kBatch) {
			double v[kBatch];
			int at[kBatch];
#pragma unroll
			for (int b = 0; b < kBatch; ++b) {
				at[b] = -1;
				if (q0 + 32 * b < total) {
					settle();
					const int2 cell = cells[e];
					const int rel = cell.y & 255, t = st - rel;
					if (t >= 0 && t < tk.nt) {
						at[b] = (sm - rel + (sm < rel ? L.depth : 0)) * L.slot + (cell.y >> 8);
						v[b] = __ldcg(tk.zeta + t * plane + cell.x);
					}
					e += 32;
				}
			}
#pragma unroll
			for (int b = 0; b < kBatch; ++b)
				if (at[b] >= 0) ring[at[b]] = v[b];
		}
		// step n's halo is waited for at the end of step n - 1, step 0's by
		// the CTA's barrier before the first
		__syncwarp();
		for (; n <= hi; ++n) {
			if (n == 0) __syncthreads();
			else bar_arrive(kBarHalo + (n - 1) % kHaloBars, kThreads);
		}
	}
}

// The publication warp: the barrier orders the compute warps' global stores of
// a step before the release store that publishes it; steps that are handed over
// meanwhile are published together.
template <int TX, int TU, int NC>
__device__ __forceinline__ void pub_warp(const Task64& tk, int bx, int c, Shared64* sh) {
	constexpr int kThreads = NC + 32;
	int* flag = tk.flags + bx * tk.nc + c;
	const int lane = threadIdx.x & 31;
	const int U0 = bx * TX + c * TU, steps = tk.nt + TU - 1;
	__syncthreads();  // step 0's halo
	for (int n = 0; n < steps;) {
		// this step, and those after it that the compute warps have left too
		const int upto = max(n + 1, min(n + kPubBars, *((volatile int*)&sh->done) - 1));
		const int last = min(__shfl_sync(0xffffffffu, upto, 0), steps);
		for (; n < last; ++n) bar_sync(kBarPub + n % kPubBars, kThreads);
		if (lane == 0) {
			*((volatile int*)&sh->published) = n;
			st_release_gpu(flag, n < steps ? U0 + n : INT_MAX);
		}
		__syncwarp();
	}
}

template <int PY, int TX, int TU>
__device__ __forceinline__ void compute_tile(const Task64& tk, int bx, int c, const Layout64& L,
                                             double* ring, const double* sphi, Shared64* sh,
                                             int* err) {
	constexpr int NC = TX * TU;
	constexpr int PYP = (PY + 1) & ~1;
	const int l = threadIdx.x % TU, xl = threadIdx.x / TU;
	const int px = tk.px, rows = tk.pt * px;
	const int x = bx * TX + xl, y = bx * TX + c * TU + l - x;
	const bool ok = x < tk.nx && y >= 0 && y < tk.ny;
	const long long plane = (long long)tk.nx * tk.ny;
	double* const z = tk.zeta + (long long)x * tk.ny + y;
	double* const own = ring + (xl + px - 1) * L.ld + l + px + PY - 2;
	unsigned own_a = static_cast<unsigned>(__cvta_generic_to_shared(own));
	unsigned taps = static_cast<unsigned>(__cvta_generic_to_shared(sphi));
	// one row up and one column left; one slot
	unsigned row_bytes = 8u * unsigned(L.ld + 1), slot_bytes = 8u * unsigned(L.slot);
	// (opaque: nothing is computed ahead for all widths of the kernel's switch)
	asm volatile("" : "+r"(own_a), "+r"(taps), "+r"(row_bytes), "+r"(slot_bytes));
	const int steps = tk.nt + TU - 1;
	int slot = l == 0 ? 0 : L.depth - l;  // of t = n - l
	double e = ok && l == 0 ? z[0] : 0.0;
	__syncthreads();  // step 0's halo
	for (int n = 0; n < steps; ++n) {
		const int t = n - l;
		// the next step's noise
		const double f = ok && t + 1 >= 0 && t + 1 < tk.nt ? z[(t + 1) * plane] : 0.0;
		double s = 0.0;
		{
			// rows of taps r = (k, i): row x-i of slice t-k
			double w[PY], p[PYP], m[PY];
			int ks = slot, i = 0;
			unsigned pa = taps, za = own_a + unsigned(ks) * slot_bytes;
			auto advance = [&] {  // to the next row
				pa += 8 * PYP;
				const bool wrap = i + 1 == px;
				i = wrap ? 0 : i + 1;
				const int kn = ks == 0 ? L.depth - 1 : ks - 1;
				ks = wrap ? kn : ks;
				za = wrap ? own_a + unsigned(ks) * slot_bytes : za - row_bytes;
			};
			// row 0's products and row 1's operands
#pragma unroll
			for (int j = 0; j < PY; ++j) w[j] = lds64(za - 8 * j);
#pragma unroll
			for (int j = 0; j < PYP; j += 2) lds128(pa + 8 * j, p[j], p[j + 1]);
			w[0] = e;  // lag (0, 0, 0): the cell's own noise
			advance();
#pragma unroll
			for (int j = 0; j < PY; ++j) {
				m[j] = mul_here(p[j], w[j]);
				w[j] = lds64(za - 8 * j);
			}
#pragma unroll
			for (int j = 0; j < PYP; j += 2) lds128(pa + 8 * j, p[j], p[j + 1]);
			// (the last two rows load rows past the last, within the ring and
			// the padding after the taps: not used)
			auto row = [&] {
				advance();
				row_step<PY>(s, m, w, p, za, pa);
			};
			// eight rows to a branch: a branch costs a lone warp about 30 cycles
			int left = rows;
			for (; left >= 8; left -= 8) {
				row();
				row();
				row();
				row();
				row();
				row();
				row();
				row();
			}
			for (; left > 0; --left) row();
		}
		s = __dadd_rn(e, s);
		const bool live = ok && t >= 0 && t < tk.nt;
		if (live) own[slot * L.slot] = s;
		// every cell of step n is in the ring, and step n + 1's halo
		if (n + 1 < steps) bar_sync(kBarHalo + n % kHaloBars, NC + 32);
		// (released before this step's global stores: it waits for none)
		if (threadIdx.x == 0) st_release_cta(&sh->done, n + 1);
		if (live) z[t * plane] = s;
		// the barrier's previous round is over once the publication warp has
		// left it (it waits for nothing but these barriers)
		for (long long it = 0; *((volatile int*)&sh->published) < n + 1 - kPubBars; ++it)
			if (it == 64ll * kSpinLimit) {
				atomicCAS(err, DEV_OK, DEV_TIMEOUT);
				break;
			}
		__syncwarp();
		bar_arrive(kBarPub + n % kPubBars, NC + 32);
		e = f;
		slot = slot + 1 == L.depth ? 0 : slot + 1;
	}
}

template <int PY, int TX, int TU>
__device__ __forceinline__ void compute_pairs(const Task64& tk, int bx, int c, const Layout64& L, double* ring,
                             const double* sphi, Shared64* sh, int* err) {
	constexpr int NC = TX / 2 * TU;
	constexpr int PYP = (PY + 1) & ~1;
	const int l = threadIdx.x % TU, rp = threadIdx.x / TU;
	const int px = tk.px, rows = tk.pt * px;
	const int x = bx * TX + 2 * rp, U0 = bx * TX + c * TU, y = U0 + l - x;
	const bool ok0 = x < tk.nx && y >= 0 && y < tk.ny;
	const bool ok1 = x + 1 < tk.nx && y - 1 >= 0 && y - 1 < tk.ny;
	const long long plane = (long long)tk.nx * tk.ny;
	double* const z0 = tk.zeta + (long long)x * tk.ny + y;
	double* const z1 = z0 + tk.ny - 1;
	double* const own = ring + (2 * rp + px - 1) * L.ld + l + px + PY - 2;
	unsigned own_a = static_cast<unsigned>(__cvta_generic_to_shared(own));
	unsigned taps = static_cast<unsigned>(__cvta_generic_to_shared(sphi));
	// one row up and one column left; one slot
	unsigned row_bytes = 8u * unsigned(L.ld + 1), slot_bytes = 8u * unsigned(L.slot);
	// (opaque: nothing is computed ahead for all widths of the kernel's switch)
	asm volatile("" : "+r"(own_a), "+r"(taps), "+r"(row_bytes), "+r"(slot_bytes));
	const int steps = tk.nt + TU - 1;
	int slot = l == 0 ? 0 : L.depth - l;  // of t = n - l
	double e0 = ok0 && l == 0 ? z0[0] : 0.0, e1 = ok1 && l == 0 ? z1[0] : 0.0;
	__syncthreads();  // step 0's halo
	for (int n = 0; n < steps; ++n) {
		const int t = n - l;
		// the next step's noise
		const bool next = t + 1 >= 0 && t + 1 < tk.nt;
		const double f0 = next && ok0 ? z0[(t + 1) * plane] : 0.0;
		const double f1 = next && ok1 ? z1[(t + 1) * plane] : 0.0;
		double s0 = 0.0, s1 = 0.0;
		{
			// Row of taps r = (k, i) at a time, both chains on the same taps:
			// chain 0 reads window r, row x-i of slice t-k, chain 1 window r-1
			// (row x+1-i) one column on; at i = 0 chain 1's row is read by
			// itself.  Two windows and two rows of taps in turn.
			double w[2][PY + 1], p[2][PYP], m0[PY], m1[PY];
			int ks = slot, i = 0;
			unsigned pa = taps, za = own_a + unsigned(ks) * slot_bytes;
			auto advance = [&] {  // to the next row; 1 at the start of a slice
				pa += 8 * PYP;
				const int start = i + 1 == px ? 1 : 0;
				i = start ? 0 : i + 1;
				const int kn = ks == 0 ? L.depth - 1 : ks - 1;
				ks = start ? kn : ks;
				za = start ? own_a + unsigned(ks) * slot_bytes : za - row_bytes;
				return start;
			};
			// row 0's products and row 1's operands
#pragma unroll
			for (int j = 0; j <= PY; ++j) {
				w[1][j] = lds64(za + row_bytes - 8 * j);
				w[0][j] = lds64(za - 8 * j);
			}
#pragma unroll
			for (int j = 0; j < PYP; j += 2) lds128(pa + 8 * j, p[0][j], p[0][j + 1]);
			w[1][1] = e1;  // lag (0, 0, 0): the cells' own noise
			w[0][0] = e0;
			int start = advance();
#pragma unroll
			for (int j = 0; j < PYP; j += 2) lds128(pa + 8 * j, p[1][j], p[1][j + 1]);
#pragma unroll
			for (int j = 0; j <= PY; ++j) {
				if (j < PY) {
					m0[j] = mul_here(p[0][j], w[0][j]);
					m1[j] = mul_here(p[0][j], w[1][j + 1]);
				}
				w[1][j] = lds64(za - 8 * j);
				if (j > 0) lds64_if(w[0][j], za + row_bytes - 8 * j, start);
			}
			// (the last two rows load rows past the last, within the ring and
			// the padding after the taps: not used)
			auto row = [&](auto odd) {
				constexpr int b = decltype(odd)::value;
				start = advance();
				pair_step<PY>(s0, s1, m0, m1, w[1 - b], w[b], p[1 - b], p[b], za, pa,
				             za + row_bytes, start);
			};
			using Even = std::integral_constant<int, 0>;
			using Odd = std::integral_constant<int, 1>;
			int left = rows;
			for (; left >= 4; left -= 4) {
				row(Even{});
				row(Odd{});
				row(Even{});
				row(Odd{});
			}
			if (left > 0) row(Even{});
			if (left > 1) row(Odd{});
			if (left > 2) row(Even{});
		}
		s0 = __dadd_rn(e0, s0);
		s1 = __dadd_rn(e1, s1);
		const bool live = t >= 0 && t < tk.nt;
		double* r = own + slot * L.slot;
		if (live && ok0) r[0] = s0;
		if (live && ok1) r[L.ld] = s1;
		// every cell of step n is in the ring, and step n + 1's halo
		if (n + 1 < steps) bar_sync(kBarHalo + n % kHaloBars, NC + 32);
		// (released before this step's global stores: it waits for none)
		if (threadIdx.x == 0) st_release_cta(&sh->done, n + 1);
		if (live && ok0) z0[t * plane] = s0;
		if (live && ok1) z1[t * plane] = s1;
		// the barrier's previous round is over once the publication warp has
		// left it (it waits for nothing but these barriers)
		for (long long it = 0; *((volatile int*)&sh->published) < n + 1 - kPubBars; ++it)
			if (it == 64ll * kSpinLimit) {
				atomicCAS(err, DEV_OK, DEV_TIMEOUT);
				break;
			}
		__syncwarp();
		bar_arrive(kBarPub + n % kPubBars, NC + 32);
		e0 = f0;
		e1 = f1;
		slot = slot + 1 == L.depth ? 0 : slot + 1;
	}
}

// POLLS: of the upstream tiles without progress before the wait gives up (a constant:
// read from the task, surfaces of few taps took 1 to 2 % longer).
template <int TX, int TU, int CELLS, int POLLS = kSpinLimit>
__global__ void __launch_bounds__(TX * TU / CELLS + 64)
ar64_tile_kernel(const Task64* __restrict__ tasks, int ntasks, int tickets,
                 int* __restrict__ counter, int* __restrict__ err) {
	constexpr int NC = TX * TU / CELLS, NTHREADS = NC + 64;
	extern __shared__ __align__(16) double smem64[];
	__shared__ Shared64 sh;
	__shared__ int s_ticket;
	const int tid = threadIdx.x;
	for (;;) {
		if (tid == 0)
			s_ticket = *((volatile int*)err) == DEV_OK ? atomicAdd(counter, 1) : tickets;
		__syncthreads();
		const int ticket = s_ticket;
		if (ticket >= tickets) return;
		int lo = 0, hi = ntasks - 1;
		while (lo < hi) {
			const int mid = (lo + hi + 1) / 2;
			if (tasks[mid].ticket_base <= ticket) lo = mid; else hi = mid - 1;
		}
		const Task64 tk = tasks[lo];
		int tile = ticket - tk.ticket_base;
		if (tk.tiles) tile = tk.tiles[tile];
		const int bx = tile / tk.nc, c = tile % tk.nc;
		const Layout64 L = layout64(TX, TU, tk.pt, tk.px, tk.py, tk.ahead);
		double* ring = smem64 + kLead;
		double* sphi = ring + size_t(L.slot) * L.depth;
		int2* cells = reinterpret_cast<int2*>(sphi + L.phi);
		const int pyp = even_up(tk.py);
		for (int q = tid; q < L.slot * L.depth; q += NTHREADS) ring[q] = 0.0;
		for (int q = tid; q < L.phi; q += NTHREADS) {
			const int j = q % pyp;
			const int row = q / pyp;
			sphi[q] = j < tk.py && row < tk.pt * tk.px ? tk.phi[row * tk.py + j] : 0.0;
		}
		if (tid == 0) {
			sh.done = 0;
			sh.published = 0;
		}
		__syncthreads();
		if (tid >= NC + 32) {
			pub_warp<TX, TU, NC>(tk, bx, c, &sh);
		} else if (tid >= NC) {
			halo_warp<TX, TU, NC, POLLS>(tk, bx, c, L, ring, cells, &sh, err);
		} else if constexpr (CELLS == 2) {
			switch (tk.py) {
#define ARMA_PY_CASE(N) case N: compute_pairs<N, TX, TU>(tk, bx, c, L, ring, sphi, &sh, err); break;
				ARMA_PY_CASE(1) ARMA_PY_CASE(2) ARMA_PY_CASE(3) ARMA_PY_CASE(4) ARMA_PY_CASE(5)
				ARMA_PY_CASE(6) ARMA_PY_CASE(7) ARMA_PY_CASE(8) ARMA_PY_CASE(9) ARMA_PY_CASE(10)
#undef ARMA_PY_CASE
				default: break;
			}
		} else {
			switch (tk.py) {
#define ARMA_PY_CASE(N) case N: compute_tile<N, TX, TU>(tk, bx, c, L, ring, sphi, &sh, err); break;
				ARMA_PY_CASE(1) ARMA_PY_CASE(2) ARMA_PY_CASE(3) ARMA_PY_CASE(4)
				ARMA_PY_CASE(5) ARMA_PY_CASE(6) ARMA_PY_CASE(7) ARMA_PY_CASE(8)
				ARMA_PY_CASE(9) ARMA_PY_CASE(10) ARMA_PY_CASE(11) ARMA_PY_CASE(12)
				ARMA_PY_CASE(13) ARMA_PY_CASE(14) ARMA_PY_CASE(15) ARMA_PY_CASE(16)
#undef ARMA_PY_CASE
				default: break;
			}
		}
		__syncthreads();
	}
}

// One launch per hyperplane, every thread the reference's truncated sum: for
// coefficients that are not finite, whose products with the tiles' zero padding
// would not vanish, and slices of 2^31 points and more.
constexpr int kPlaneThreads = 128;
__global__ void __launch_bounds__(kPlaneThreads)
ar64_plane_kernel(double* __restrict__ zeta, const double* __restrict__ phi,
                  int nt, int nx, int ny, int pt, int px, int py, int s, int t_lo) {
	const int t = t_lo + blockIdx.y;
	const int rem = s - t;                 // x + y
	const int x_lo = max(0, rem - (ny - 1));
	const int x = x_lo + blockIdx.x * kPlaneThreads + threadIdx.x;
	const int x_hi = min(nx - 1, rem);
	if (t >= nt || x > x_hi) return;
	const int y = rem - x;
	const long long sx = ny, st = (long long)nx * ny;
	const int m1 = min(t + 1, pt), m2 = min(x + 1, px), m3 = min(y + 1, py);
	double sum = 0.0;
	for (int k = 0; k < m1; ++k) {
		for (int i = 0; i < m2; ++i) {
			const double* prow = phi + (k * px + i) * py;
			const double* zrow = zeta + (t - k) * st + (x - i) * sx + y;
			for (int j = 0; j < m3; ++j)
				sum = __dadd_rn(sum, __dmul_rn(prow[j], zrow[-j]));
		}
	}
	double* p = zeta + t * st + x * sx + y;
	*p = __dadd_rn(*p, sum);
}

void launch_planes(Ctx* c, const Ar64Surface& s) {
	for (int q = 0; q < s.nt + s.nx + s.ny - 2; ++q) {
		const int t_lo = std::max(0, q - (s.nx - 1) - (s.ny - 1));
		const int t_hi = std::min(s.nt - 1, q);
		const int xs = std::min(s.nx, q + 1);
		// the launch's second dimension holds at most 65535 slices
		for (int t = t_lo; t <= t_hi; t += 65535) {
			const dim3 grid((xs + kPlaneThreads - 1) / kPlaneThreads,
			                std::min(t_hi - t + 1, 65535));
			ar64_plane_kernel<<<grid, kPlaneThreads, 0, c->stream>>>(
			    s.zeta, s.phi, s.nt, s.nx, s.ny, s.pt, s.px, s.py, q, t);
			ARMA_CUDA_TRY(cudaGetLastError());
			c->launches += 1;
		}
	}
}

// Whether the tiles take a surface: finite coefficients, offsets in a slice of 32 bits.
bool by_tiles(const Ar64Surface& s) {
	return s.finite && (long long)s.nx * s.ny <= INT_MAX;
}

// The halo steps a tile of this shape can keep ahead; 0: it does not fit.
int ahead_of(int tx, int tu, const Ar64Surface& s) {
	for (int a = kMaxAhead; a > 0; --a)
		if (layout64(tx, tu, s.pt, s.px, s.py, a).bytes <= kSmemLimit) return a;
	return 0;
}

// A surface's tiles by anti-diagonals (2 bx + c ascending): the tiles that a tile's
// halo comes from (bx, c - 1 and c - 2; bx - 1, c - 1 to c + 1) come before it.
void diagonal_order(int nbx, int nc, int* list) {
	for (int key = 0; key <= 2 * (nbx - 1) + nc - 1; ++key)
		for (int b = std::max(0, (key - nc + 2) / 2); b < nbx && 2 * b <= key; ++b)
			*list++ = b * nc + key - 2 * b;
}

int tiles_per_row(int tx, int tu, int ny) { return (ny + tx - 1 + tu - 1) / tu; }

template <int TX, int TU, int CELLS>
void launch_tiles(Ctx* c, std::vector<Ar64Surface> surfs) {
	// longest dependency chains first
	auto chain = [](const Ar64Surface& s) {
		return double(s.nt + s.nx + s.ny) * s.pt * s.px * s.py;
	};
	std::stable_sort(surfs.begin(), surfs.end(), [&](const Ar64Surface& a, const Ar64Surface& b) {
		return chain(a) > chain(b);
	});
	std::vector<Task64> tasks;
	long long tickets = 0;
	size_t smem = 0;
	for (const Ar64Surface& s : surfs) {
		Task64 t;
		t.nt = s.nt; t.nx = s.nx; t.ny = s.ny;
		t.pt = s.pt; t.px = s.px; t.py = s.py;
		t.nbx = (s.nx + TX - 1) / TX;
		t.nc = tiles_per_row(TX, TU, s.ny);
		t.ticket_base = int(tickets);
		t.ahead = ahead_of(TX, TU, s);
		t.zeta = s.zeta;
		t.phi = s.phi;
		t.flags = nullptr;
		tickets += (long long)t.nbx * t.nc;
		ARMA_REQUIRE(tickets < INT_MAX / 4, ARMA_EINVAL, "surface too large");
		smem = std::max(smem, layout64(TX, TU, s.pt, s.px, s.py, t.ahead).bytes);
		tasks.push_back(t);
	}
	// step counters of every tile, then the ticket counter
	int* flags = static_cast<int*>(scratch_take(c, sizeof(int) * (size_t(tickets) + 1)));
	ARMA_CUDA_TRY(cudaMemsetAsync(flags, 0, sizeof(int) * (size_t(tickets) + 1), c->stream));
	constexpr int threads = TX * TU / CELLS + 64;
	auto kernel = ar64_tile_kernel<TX, TU, CELLS>;
	ARMA_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
	                                   int(kSmemLimit)));
	int per_sm = 0;
	ARMA_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem));
	ARMA_REQUIRE(per_sm > 0, ARMA_EINVAL, "AR tile does not fit in shared memory");
	const int grid = int(std::min<long long>(tickets, (long long)per_sm * c->num_sms));
	// Where the tiles do not all run at once they are handed out by anti-diagonals:
	// row by row, the CTAs hold a band of tile rows end to end, and a surface of few
	// slices is swept once per band (ms, row by row / by anti-diagonals: 1 x 1000 x
	// 1000 of order 1 x 16 x 1 51.7 / 10.1, 16 x 500 x 500 of 10^3 28.2 / 13.7, 200^3 of
	// 10^3 7.7 / 6.7; all at once, 64 x 30 x 1000 of 3 x 6 x 6 2.24 / 2.41).
	int* d_tiles = nullptr;
	std::vector<int> tiles;
	if (tickets > grid) {
		tiles.resize(size_t(tickets));
		for (const Task64& t : tasks) diagonal_order(t.nbx, t.nc, tiles.data() + t.ticket_base);
		d_tiles = static_cast<int*>(scratch_take(c, sizeof(int) * tiles.size()));
		ARMA_CUDA_TRY(copy_async(c, d_tiles, tiles.data(), sizeof(int) * tiles.size(),
		                         cudaMemcpyHostToDevice, c->stream));
	}
	for (Task64& t : tasks) {
		t.flags = flags + t.ticket_base;
		t.tiles = d_tiles ? d_tiles + t.ticket_base : nullptr;
	}
	auto* d_tasks = static_cast<Task64*>(scratch_take(c, sizeof(Task64) * tasks.size()));
	ARMA_CUDA_TRY(copy_async(c, d_tasks, tasks.data(), sizeof(Task64) * tasks.size(),
	                         cudaMemcpyHostToDevice, c->stream));
	kernel<<<grid, threads, smem, c->stream>>>(d_tasks, int(tasks.size()), int(tickets),
	                                           flags + tickets, c->d_err);
	ARMA_CUDA_TRY(cudaGetLastError());
	c->launches += 1;
}

}  // namespace

void launch_ar64(Ctx* c, const std::vector<Ar64Surface>& surfaces) {
	ProfScope prof_(c, "ar64");
	// Tile shapes, by how many cells can be at work at once if none waits for an
	// SM (all steps of all tiles over the longest chain).  16 x 16 by pairs moves
	// the most cells per cycle and is the slowest step (21 cycles a tap): taken
	// where more than 96 cells per SM are at work.  8 x 16 (14 cycles a tap) below
	// that, 4 x 16 (11) where all its tiles have an SM to themselves.  Measured (tiles
	// row by row), 16 x 16 / 8 x 16 / 4 x 16 (ms): 40 cells per SM 3.9 / 2.7 / 3.1; 79 (400 x 128 x
	// 128 of order 10^3) 7.0 / 4.9 / 5.5; 108 3.7 / 4.4 / 4.6; 142 10.1 / 10.9 /
	// 12.1; 415 (16 mixed surfaces) 10.2 / 13.7 / 17.5; 200 x 40 x 40 alone, 30 tiles
	// of 4 x 16, 1.14 / 0.76 / 0.65.  8 x 16 too for rows of more taps than a pair's
	// registers hold, 4 x 16 and 8 x 8 for orders whose ring does not fit otherwise.
	std::vector<Ar64Surface> groups[4];
	long long t4 = 0;
	double work = 0, chain = 0;
	for (const Ar64Surface& s : surfaces)
		if (by_tiles(s)) {
			const double taps = double(s.pt) * s.px * s.py;
			t4 += (long long)((s.nx + 3) / 4) * tiles_per_row(4, 16, s.ny);
			work += 256.0 * ((s.nx + 15) / 16) * tiles_per_row(16, 16, s.ny) * (s.nt + 15) * taps;
			chain = std::max(chain, (double(s.nt) + s.nx + s.ny) * taps);
		}
	const int want = t4 <= c->num_sms ? 2 : work <= 96.0 * c->num_sms * chain ? 1 : 0;
	for (const Ar64Surface& s : surfaces) {
		if (!by_tiles(s)) launch_planes(c, s);
		else if (want == 0 && s.py <= kPairTaps && ahead_of(16, 16, s)) groups[0].push_back(s);
		else if (want <= 1 && ahead_of(8, 16, s)) groups[1].push_back(s);
		else if (ahead_of(4, 16, s)) groups[2].push_back(s);
		else groups[3].push_back(s);
	}
	if (!groups[0].empty()) launch_tiles<16, 16, 2>(c, groups[0]);
	if (!groups[1].empty()) launch_tiles<8, 16, 1>(c, groups[1]);
	if (!groups[2].empty()) launch_tiles<4, 16, 1>(c, groups[2]);
	if (!groups[3].empty()) launch_tiles<8, 8, 1>(c, groups[3]);
}

void launch_ar64_starved(Ctx* c) {
	constexpr int TX = 8, TU = 16;
	const size_t cells = 2 * size_t(TX) * TU;
	auto* zeta = static_cast<double*>(scratch_take(c, sizeof(double) * (cells + 2)));
	int* flags = static_cast<int*>(scratch_take(c, sizeof(int) * 3));
	ARMA_CUDA_TRY(cudaMemsetAsync(zeta, 0, sizeof(double) * (cells + 2), c->stream));
	Task64 t{};
	t.nt = 2; t.nx = TX; t.ny = TU;
	t.pt = t.px = 1; t.py = 2;
	t.nbx = 1;
	t.nc = tiles_per_row(TX, TU, TU);  // 2
	t.ahead = 1;
	t.zeta = zeta;
	t.phi = zeta + cells;
	t.flags = flags;
	auto* d_task = static_cast<Task64*>(scratch_take(c, sizeof(Task64)));
	const int start[3] = {0, 0, 1};  // nothing done; the next ticket: the second tile
	ARMA_CUDA_TRY(copy_async(c, d_task, &t, sizeof(t), cudaMemcpyHostToDevice, c->stream));
	ARMA_CUDA_TRY(copy_async(c, flags, start, sizeof(start), cudaMemcpyHostToDevice, c->stream));
	const size_t smem = layout64(TX, TU, t.pt, t.px, t.py, t.ahead).bytes;
	auto kernel = ar64_tile_kernel<TX, TU, 1, kStarvedPolls>;
	ARMA_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
	                                   int(kSmemLimit)));
	ProfScope prof_(c, "ar64");
	kernel<<<1, TX * TU + 64, smem, c->stream>>>(d_task, 1, t.nc, flags + 2, c->d_err);
	ARMA_CUDA_TRY(cudaGetLastError());
	c->launches += 1;
}

}  // namespace armab
