// FP32 compensated AR filter: a persistent tile wavefront over a batch of
// independent surfaces.
//
// The filter (reference src/generator/ar_model_surf.cc:5-36) is
//     zeta(t,x,y) = eps(t,x,y) + sum_{(k,i,j) != 0} phi(k,i,j) zeta(t-k,x-i,y-j)
// with zeta = 0 outside the array.  Because phi(0,i,j) != 0, every point
// depends on earlier points of its own time slice as well as on the previous
// pt-1 slices.  The work is split into spatial tiles of TX x TY points; one
// CTA owns one tile of one surface for all t and walks the slices in order.
// For slice t its four compute warps
//   1. accumulate the terms on slices t-1 .. t-pt+1 (90% of the work for a
//      10^3 model) from a shared-memory ring that holds those slices for the
//      tile plus its west/north halo,
//   2.-3. wait for slice t's halo, which a fifth warp brings in a slice ahead
//      (slot t cleared, the three neighbour tiles x-1, y-1 and both seen to
//      have published slice t, their values copied; bounded polls of a
//      per-tile counter in global memory), and add the current-slice terms
//      that reach into it (the in-tile part of the current slice is held at
//      zero),
//   4. solve the remaining in-tile recursion zeta = S + A0 zeta exactly as a
//      quarter-plane convolution zeta = H * S, where H is the impulse response
//      of 1 / (1 - A0(z1,z2)) on the tile (precomputed in FP64),
//   5. store the slice to the ring and to global memory; the fifth warp
//      publishes it (release store after a barrier) off the compute warps'
//      critical path.
// The ring has one slot more than the slices in use, so that the halo of slice
// t+1 comes in while slice t is computed (512 x 256 x 256 points of order 10^3,
// one tile per SM: 5.42 -> 5.20 ms; the batch of 256 surfaces 52.3 -> 51.8 ms;
// one 64 x 32 x 32 surface 258 -> 241 us); the largest orders can go without it
// (launch_ar32c).
// The coefficients are carried as hi + lo float pairs (rounding phi to one
// float perturbs a high-gain recursion far more than FP32 summation does):
// each (k,i) row of taps feeds two FP32 FMA chains over one register window,
// the two of an output side by side in one packed FMA (fma.rn.f32x2, each half
// rounded as fmaf: half the instructions), continued across the rows of one k
// plane, and the plane totals are combined
// with Kahan compensation (per row, the compensation cost 7 % more time for
// 0.2-1.2e-6 less RMS error).  H is applied in plain FP32, one FMA chain per
// output over up to three rows of H (up to 96 taps), the at most six chain
// totals of an output Kahan-added: it acts once per slice on the current
// slice alone, and its rounding changes the surface by far less than phi's (a
// lo part for H moved the RMS error by under 1e-7 at 18 % of the filter's
// time; Kahan-adding every row of H instead of every three rows, by 4e-8 at
// 5 %).  Tiles are handed out through a global ticket
// counter in dependency order, so a CTA only ever waits on tiles that are
// already owned by running CTAs.
//
// Bound by the issue slots and latencies of 12 compute warps per SM (with one
// FMA per chain: FMA pipe 47 % busy, issue 66 %, shared-memory loads half).
// Packed FMAs, one copy of the tap loop for all k, 16-byte accesses of noise, S
// and results, and the H units numbered so that neighbouring lanes read the same
// rows of H: the batch of 256 surfaces 51.7 -> 48.2 ms, 512 x 256 x 256 alone
// 5.20 -> 5.06, 64 x 32 x 32 241 -> 217 us.  Without the packed FMAs the batch
// took 52.4 ms, with the Kahan steps packed too 49.5; two rows of taps at once
// cost 4 % (the code of several tap counts on an SM outgrows its instruction
// cache).
#include <algorithm>
#include <climits>
#include <cmath>
#include <mutex>
#include <type_traits>
#include <vector>

#include "internal.h"

namespace armab {
namespace {

constexpr int TX = 16;            // tile rows (x)
constexpr int TY = 32;            // tile columns (y)
constexpr int R = 8;              // outputs per thread along y
constexpr int STRIPS = TY / R;    // threads per tile row
constexpr int GROUP = TX * STRIPS; // threads covering the tile once
constexpr int NCOMP = 2 * GROUP;   // compute threads: two groups split the tap rows
constexpr int NTHREADS = NCOMP + 32; // plus the halo / publication warp
// named barriers (0 is __syncthreads)
constexpr int BAR_HALO = 1;        // (2, by slice parity) halo warp -> compute: halo of t in slot t
constexpr int BAR_COMP = 3;        // compute threads among themselves
constexpr int BAR_PUB = 4;         // (PUB_BARS, by slice) compute -> halo warp: slice t stored
constexpr int PUB_BARS = 8;
constexpr int LH = 12;            // left (y) halo columns held in the ring
constexpr int W = LH + TY;        // ring row width (floats)
constexpr int SPAD = TY + 8;      // zero padding left of each S row
constexpr int SW = SPAD + TY + 4; // S row width (padded against bank conflicts)
constexpr int MAXO = 13;          // max order per axis supported (py <= LH+1)
constexpr int HS = TY + 4;        // H row stride in shared memory (bank spread)
constexpr int HCH = 3;            // rows of H per H work unit
constexpr int HPAIR = 51;         // H work units per strip pair: sum_x ceil((x+1)/HCH)
constexpr int HUNITS = 2 * HPAIR; // H work units per tile slice (<= NCOMP)
constexpr int PS = 2 * R + 4;     // partial record stride (bank spread)
static_assert(TX == 16 && TY == 4 * R && HUNITS <= NCOMP, "H work-unit table assumes 16 x 4R tiles");
constexpr int kMaxTapRows = MAXO * (TX + 1);  // (k, i) tap rows per model: pt * px
constexpr int kSpinLimit = 1 << 24;
constexpr int kAheadPolls = 1 << 12;
constexpr int kAhead = 2;          // slices, where tiles keep pace
constexpr int kHeavyTaps = 400;    // taps whose tiles crowd each other out on an SM

struct Task {
	int nt, nx, ny, pt, px, py;
	int t0;  // slices [0, t0) are history: read, never written
	int given_tx : 29;  // tile rows [0, given_tx) are given (an x-strip's upper band): read, never written
	unsigned lead : 1;  // slices that the halo comes in ahead; 0: no slot of the ring for it
	unsigned pace : 1;  // tiles run at most kAhead slices ahead of the tiles below them
	unsigned diagonal : 1;  // tiles handed out by anti-diagonals, else row by row
	int tiles_x, tiles_y;
	int ticket_base;
	int polls;  // of the neighbours without progress before the wait gives up
	float* zeta;
	const float* phi;     // hi part, pt*px*py
	const float* phi_lo;  // lo part: phi - hi, pt*px*py
	const float* h;       // intra-slice response, TX*TY
	int* flags;
};

__device__ __forceinline__ void kahan_add(float& s, float& c, float v) {
	const float y = v - c;
	const float t = s + y;
	c = (t - s) - y;
	s = t;
}

// a pair of floats in one 64-bit register pair
__device__ __forceinline__ unsigned long long pack2(float a, float b) {
	unsigned long long v;
	asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
	return v;
}

__device__ __forceinline__ float2 unpack2(unsigned long long v) {
	float2 r;
	asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
	return r;
}

// (c.x + a.x b.x, c.y + a.y b.y), each half rounded as fmaf
__device__ __forceinline__ void fma2(unsigned long long& c, unsigned long long a,
                                     unsigned long long b) {
	asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}

__device__ __forceinline__ void cp_async16(float* dst_smem, const float* src) {
	const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst_smem));
	asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}

__device__ __forceinline__ void bar_sync(int id, int n) {
	asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory");
}

__device__ __forceinline__ void bar_arrive(int id, int n) {
	asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory");
}

__device__ __forceinline__ void cp_async_wait_all() {
	asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

__device__ __forceinline__ int ld_acquire(const int* p) {
	int v;
	asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
	return v;
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

__device__ __forceinline__ void st_release(int* p, int v) {
	asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Whether every non-null flag is >= need; the three acquire loads of a poll are
// issued together so one L2 round trip covers them.  seen[] holds the values
// this thread's earlier acquire loads returned: a neighbour that is already
// known to be at or past `need` is not polled again (that load's acquire already
// ordered its slices before this thread's later loads), so a tile whose
// neighbours run ahead pays no round trip.
__device__ bool flags_reached(const int* f0, const int* f1, const int* f2, int need, int* seen) {
	if (seen[0] >= need && seen[1] >= need && seen[2] >= need) return true;
	const int a = f0 ? ld_acquire(f0) : need;
	const int b = f1 ? ld_acquire(f1) : need;
	const int c = f2 ? ld_acquire(f2) : need;
	seen[0] = f0 ? a : INT_MAX;
	seen[1] = f1 ? b : INT_MAX;
	seen[2] = f2 ? c : INT_MAX;
	return a >= need && b >= need && c >= need;
}

// zeta = H * S over the quarter plane of one tile, cut into work units of
// equal cost.  Row x of the output needs the x+1 rows dx = 0..x of H, each a
// causal 1-D convolution along y; the four 8-column strips of a row cost 1, 2,
// 3 and 4 blocks of R x R taps (the first block of each a triangle), so the
// strips are paired (3, 0) and (2, 1): either pair costs two triangles and
// three full blocks per row of H.  A unit is one strip pair of one output row
// over at most HCH consecutive rows of H; units are numbered pair-major, then by
// chunk c of HCH rows of H, then by output row (chunk c has the rows x >= HCH c),
// so neighbouring lanes read the same row of H and rows of S that are SW floats
// apart, whose 16-byte loads fall in different banks.  Unit u writes its partial
// (strip X in slots 0..R-1, strip Y in R..2R-1), one plain FP32 FMA chain per
// output, to part[u * PS ..]; the partials of an output are Kahan-added
// afterwards.  The unit is inlined into every tap-count instantiation of
// compute_tile: as a call, the registers the caller keeps across it spilled, and
// the filter ran 7 % slower; one copy for all of them, between switches over the
// tap count, ran 2 to 8 % slower.
// h_start: the first unit of chunk c within its pair.
__device__ __forceinline__ int h_start(int c) { return TX * c - HCH * c * (c - 1) / 2; }

// Unit u of the numbering: its strip pair, output row and rows of H.
struct HUnit {
	int pair, x, dx0, dx1;
};

__device__ __forceinline__ HUnit h_unit_of(int u) {
	HUnit h;
	h.pair = u >= HPAIR ? 1 : 0;
	const int v = u - h.pair * HPAIR;
	int c = 0;
	while (h_start(c + 1) <= v) ++c;
	h.x = HCH * c + v - h_start(c);
	h.dx0 = HCH * c;
	h.dx1 = min(h.dx0 + HCH, h.x + 1);
	return h;
}

__device__ __forceinline__ void load_row(float* d, const float* s, int n4) {
#pragma unroll 4
	for (int q = 0; q < n4; ++q) {
		const float4 v = reinterpret_cast<const float4*>(s)[q];
		d[4 * q] = v.x;
		d[4 * q + 1] = v.y;
		d[4 * q + 2] = v.z;
		d[4 * q + 3] = v.w;
	}
}

// acc[r] += sum_dd hv[dd] src[R + r - dd]: one full R x R block of taps
__device__ __forceinline__ void h_block(float* acc, const float* src, const float* hrow) {
	float w[2 * R], hv[R];
	load_row(w, src, 2 * R / 4);
	load_row(hv, hrow, R / 4);
#pragma unroll
	for (int r = 0; r < R; ++r) {
#pragma unroll
		for (int dd = 0; dd < R; ++dd) acc[r] = fmaf(hv[dd], w[R + r - dd], acc[r]);
	}
}

__device__ __forceinline__ void h_unit(const float* ss, const float* sh, const HUnit& h, int u,
                                       float* part) {
	const int pair = h.pair, x = h.x, dx0 = h.dx0, dx1 = h.dx1;
	const int yx = pair ? 2 * R : 3 * R;  // first column of strip X
	const int yy = pair ? R : 0;          // first column of strip Y
	const int w3 = pair ? 0 : 2 * R;      // sources of the third block
	// one FMA chain per output over the unit's rows of H
	float pX[R], pY[R];
#pragma unroll
	for (int r = 0; r < R; ++r) { pX[r] = 0.0f; pY[r] = 0.0f; }
	for (int dx = dx0; dx < dx1; ++dx) {
		const float* srow = ss + (x - dx) * SW + SPAD;
		const float* hrow = sh + dx * HS;
		float wt[R], hv[R];
		// triangle of strip X: its block dy0 = yx reaches sources srow[0 .. r]
		load_row(wt, srow, R / 4);
		load_row(hv, hrow + yx, R / 4);
#pragma unroll
		for (int r = 0; r < R; ++r) {
#pragma unroll
			for (int dd = 0; dd <= r; ++dd) pX[r] = fmaf(hv[dd], wt[r - dd], pX[r]);
		}
		// strip X's blocks dy0 = yx - R and yx - 2R
		h_block(pX, srow, hrow + yx - R);
		h_block(pX, srow + R, hrow + yx - 2 * R);
		// third block: strip 3's dy0 = 0 (pair 0) or strip 1's dy0 = 0 (pair 1)
		float q[R];
#pragma unroll
		for (int r = 0; r < R; ++r) q[r] = pair ? pY[r] : pX[r];
		h_block(q, srow + w3, hrow);
#pragma unroll
		for (int r = 0; r < R; ++r) {
			pX[r] = pair ? pX[r] : q[r];
			pY[r] = pair ? q[r] : pY[r];
		}
		// triangle of strip Y
		load_row(hv, hrow + yy, R / 4);
#pragma unroll
		for (int r = 0; r < R; ++r) {
#pragma unroll
			for (int dd = 0; dd <= r; ++dd) pY[r] = fmaf(hv[dd], wt[r - dd], pY[r]);
		}
	}
	float* out = part + u * PS;
#pragma unroll
	for (int q4 = 0; q4 < R / 4; ++q4) {
		reinterpret_cast<float4*>(out)[q4] =
		    make_float4(pX[4 * q4], pX[4 * q4 + 1], pX[4 * q4 + 2], pX[4 * q4 + 3]);
		reinterpret_cast<float4*>(out + R)[q4] =
		    make_float4(pY[4 * q4], pY[4 * q4 + 1], pY[4 * q4 + 2], pY[4 * q4 + 3]);
	}
}

// Layout of a tile's shared memory (floats).
struct Layout {
	int hx, slot_sz, slots;   // halo rows, floats per ring slot, ring slots
	int taps;                 // coefficients (rows of PYP)
	int pyp;
};

__host__ __device__ inline Layout tile_layout(int pt, int px, int py, int lead) {
	Layout l;
	l.hx = px - 1;
	l.slot_sz = (TX + px - 1) * W;
	l.slots = pt + lead;  // the pt slices in use and the next one's halo
	l.pyp = (py + 3) & ~3;
	l.taps = pt * px * l.pyp;
	return l;
}

// The slices that both tiles below (x + 1, y + 1) have published; t where none has
// published any: a tile that is not yet at work holds nobody back.
__device__ int slices_below(const int* fE, const int* fS, int t) {
	const int e = fE ? *((volatile const int*)fE) : 0, s = fS ? *((volatile const int*)fS) : 0;
	return e > 0 && s > 0 ? min(e, s) : e + s > 0 ? e + s : t;
}

// Where the two sides of a CTA stand on the current tile.
struct Progress {
	int done;       // slices finished by the compute warps
	int published;  // slices taken over for publication
};

// The halo / publication warp takes whichever of its two tasks is ready,
// both off the compute warps' path:
//   publish: a barrier orders the compute warps' global stores of the
//   slices they have finished before the release store of the count;
//   halo, a slice ahead of them: once slice t-2 is done (the last to
//   read the old contents of slot t; t-1 in a ring of pt slots) it clears
//   slot t and, when the three neighbour tiles have published slice t,
//   loads slice t's halo.
// Waiting for the neighbours runs out after the task's polls without progress:
// the error word is set, the tile runs on without its halo, and the call fails.
// A tile that keeps pace, more than kAhead slices ahead of the tiles below it, also
// holds back its next halo, for kAheadPolls polls at most: it waits for nobody, it gives way.
template <bool BY_TASK>
__device__ __noinline__ void halo_warp(const Task& tk, int bx, int by, const Layout& L, float* ring,
                                       Progress* sh, int* err) {
	const int lane = threadIdx.x & 31;
	const int hx = L.hx, slot_sz = L.slot_sz, slots = L.slots;
	const int x0 = bx * TX, y0 = by * TY;
	const long long sst = (long long)tk.nx * tk.ny;
	// 16-byte halo chunks need 16-byte aligned rows in global memory
	const bool vec_ok = (tk.ny % 4 == 0) &&
	                    ((reinterpret_cast<uintptr_t>(tk.zeta) & 15) == 0) && ((sst % 4) == 0);
	const int* fW = (bx > 0) ? tk.flags + (bx - 1) * tk.tiles_y + by : nullptr;
	const int* fN = (by > 0) ? tk.flags + bx * tk.tiles_y + by - 1 : nullptr;
	const int* fNW = (bx > 0 && by > 0) ? tk.flags + (bx - 1) * tk.tiles_y + by - 1 : nullptr;
	int* own_flag = tk.flags + bx * tk.tiles_y + by;
	const int* fE = by + 1 < tk.tiles_y ? own_flag + 1 : nullptr;
	const int* fS = bx + 1 < tk.tiles_x ? own_flag + tk.tiles_y : nullptr;
	int seen[3] = {-1, -1, -1};
	const bool pace = BY_TASK && tk.pace;
	const int lead = BY_TASK ? tk.lead : 1;
	int below = 0;              // slices that the tiles below have published
	int pub = tk.t0;            // slices published
	int t = tk.t0;              // the next slice to bring the halo of
	bool cleared = false;       // slot t
	long long idle = 0;
	while (pub < tk.nt) {
		const int done = __shfl_sync(0xffffffffu, lane == 0 ? ld_acquire_cta(&sh->done) : 0, 0);
		if (done > pub) {
			for (; pub < done; ++pub) bar_sync(BAR_PUB + pub % PUB_BARS, NTHREADS);
			if (lane == 0) {
				*((volatile int*)&sh->published) = pub;
				st_release(own_flag, pub);
			}
			__syncwarp();
			idle = 0;
		}
		if (t >= tk.nt || done < t - lead) {
			++idle;  // the compute warps are at work: they end every slice
			if (idle > 64ll * kSpinLimit) {
				if (lane == 0) atomicExch(err, DEV_TIMEOUT);
				break;
			}
			__nanosleep(100);
			continue;
		}
		float* cur = ring + (t % slots) * slot_sz;
		if (!cleared) {
			for (int q = lane; q < slot_sz / 4; q += 32)
				reinterpret_cast<float4*>(cur)[q] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
			__syncwarp();
			cleared = true;
		}
		int ok = 1;
		if (lane == 0) {
			ok = flags_reached(fW, fN, fNW, t + 1, seen) ? 1 : 0;
			if (pace && ok && t > below + kAhead && idle < kAheadPolls) {
				below = slices_below(fE, fS, t);
				ok = t <= below + kAhead;
			}
			if (!ok && (idle & 63) == 63 && *((volatile int*)err) != DEV_OK) ok = 1;
			if (!ok && idle > tk.polls) {
				atomicExch(err, DEV_TIMEOUT);
				ok = 1;
			}
		}
		ok = __shfl_sync(0xffffffffu, ok, 0);
		if (!ok) {
			++idle;
			__nanosleep(32);
			continue;
		}
		idle = 0;
		// rows above the tile (all columns) and the left columns of the
		// tile rows, in 16-byte chunks copied with L2-only asynchronous
		// copies (scalar loads at ragged edges)
		const float* zt = tk.zeta + t * sst;
		const int top = hx * (W / 4);
		const int nch = top + TX * (LH / 4);
		for (int q = lane; q < nch; q += 32) {
			int rr, c4;
			if (q < top) {
				rr = q / (W / 4);
				c4 = q % (W / 4);
			} else {
				rr = hx + (q - top) / (LH / 4);
				c4 = (q - top) % (LH / 4);
			}
			const int x = x0 - hx + rr, y = y0 - LH + 4 * c4;
			if (x < 0 || x >= tk.nx) continue;  // stays zero
			float* dst = cur + rr * W + 4 * c4;
			const float* src = zt + (long long)x * tk.ny + y;
			if (vec_ok && y >= 0 && y + 4 <= tk.ny) {
				cp_async16(dst, src);
			} else {
				for (int e = 0; e < 4; ++e)
					if (y + e >= 0 && y + e < tk.ny) dst[e] = __ldcg(src + e);
			}
		}
		cp_async_wait_all();
		__syncwarp();
		bar_arrive(BAR_HALO + (t & 1), NTHREADS);
		++t;
		cleared = false;
	}
}

template <int PY>
__device__ __forceinline__ void compute_tile(const Task& tk, int bx, int by, const Layout& L,
                                             float* smem, const unsigned char* s_lo, Progress* sh,
                                             int* err) {
	const int tid = threadIdx.x;
	const int grp = tid / GROUP;                 // 0 or 1: halves of the tap rows
	const int lt = tid % GROUP;
	const int xl = lt / STRIPS;                  // tile-local row
	const int yl0 = (lt % STRIPS) * R;           // tile-local first column
	const int pt = tk.pt, px = tk.px;
	const int hx = L.hx, slot_sz = L.slot_sz, slots = L.slots;
	constexpr int PYP = (PY + 3) & ~3;           // padded tap row
	const int x0 = bx * TX, y0 = by * TY;
	const long long sst = (long long)tk.nx * tk.ny;

	float* ring = smem;                          // slots
	float* sphi = ring + slots * slot_sz;        // (hi, lo) pairs
	float* sh_h = sphi + 2 * L.taps;             // TX*HS
	float* ss = sh_h + TX * HS;                  // TX*SW
	float* part = ss + TX * SW;                  // HUNITS*PS: H-unit partials
	float* comb = part;                          // GROUP*R: group 1 partials (before H)
	const int gx = x0 + xl;

	bool all_lo = true;  // no row skips its lo chain
	for (int q = 0; q < pt * px; ++q) all_lo = all_lo && s_lo[q];
	const HUnit hu = h_unit_of(min(tid, HUNITS - 1));  // found once, not per slice
	// 16-byte pieces of the tile's rows in global memory
	const bool vec = tk.ny % 4 == 0 && (reinterpret_cast<uintptr_t>(tk.zeta) & 15) == 0;
	int st = tk.t0 % slots;  // slot of slice t
	for (int t = tk.t0; t < tk.nt; ++t, st = st + 1 == slots ? 0 : st + 1) {
		float* cur = ring + st * slot_sz;
		float* zt = tk.zeta + t * sst;
		// group 0 starts from the noise of its strip (own tile: written by an
		// earlier kernel), group 1 from zero
		float s[R], c[R];
#pragma unroll
		for (int r = 0; r < R; ++r) s[r] = c[r] = 0.0f;
		if (grp == 0 && gx < tk.nx) {
			const float* zn = zt + (long long)gx * tk.ny + y0 + yl0;
			if (vec) {
#pragma unroll
				for (int q = 0; q < R / 4; ++q)
					if (y0 + yl0 + 4 * q < tk.ny) {
						const float4 v = reinterpret_cast<const float4*>(zn)[q];
						s[4 * q] = v.x;
						s[4 * q + 1] = v.y;
						s[4 * q + 2] = v.z;
						s[4 * q + 3] = v.w;
					}
			} else {
#pragma unroll
				for (int r = 0; r < R; ++r)
					if (y0 + yl0 + r < tk.ny) s[r] = zn[r];
			}
		}
		// 1. the planes of slices t-1, t-2, ..; 2./3. slot t cleared, the
		// neighbours' slice t published and its halo loaded, plane 0
		const int np = min(pt - 1, t);
		for (int m = 0, sk = st; m <= np; ++m) {
			const bool last = m == np;
			const int k = last ? 0 : m + 1;
			if (last) {
				bar_sync(BAR_HALO + (t & 1), NTHREADS);
				sk = st;
			} else {
				sk = sk == 0 ? slots - 1 : sk - 1;
			}
			// One (k, i) row of taps at a time, rows alternating between the two
			// groups: the chains of the hi and lo parts run across the rows of the
			// plane, whose total is Kahan-added to the running sum.
			const float* zb = ring + sk * slot_sz + (xl + hx) * W + yl0;
			const float* prow = sphi + (k * px) * 2 * PYP;
			unsigned long long pq[R];
#pragma unroll
			for (int r = 0; r < R; ++r) pq[r] = 0ull;
			auto rows = [&](auto every) {
#pragma unroll 1
				for (int i = (k * px + grp) & 1; i < px; i += 2) {
					const float* zr = zb - i * W;
					float win[R + LH];
#pragma unroll
					for (int q = 0; q < (R + LH) / 4; ++q) {
						const float4 v = reinterpret_cast<const float4*>(zr)[q];
						win[4 * q] = v.x;
						win[4 * q + 1] = v.y;
						win[4 * q + 2] = v.z;
						win[4 * q + 3] = v.w;
					}
					unsigned long long ph[PYP];
#pragma unroll
					for (int q = 0; q < PYP / 2; ++q) {
						const ulonglong2 v = reinterpret_cast<const ulonglong2*>(prow + i * 2 * PYP)[q];
						ph[2 * q] = v.x;
						ph[2 * q + 1] = v.y;
					}
					if (every.value || s_lo[k * px + i]) {  // warp-uniform
						// by element of the window, last first: taps ascending per output
#pragma unroll
						for (int q = R + PY - 2; q >= 0; --q) {
							const float w = win[LH - PY + 1 + q];
							const unsigned long long ww = pack2(w, w);
#pragma unroll
							for (int r = 0; r < R; ++r) {
								const int j = r - q + PY - 1;
								if (j >= 0 && j < PY) fma2(pq[r], ph[j], ww);
							}
						}
					} else {
#pragma unroll
						for (int r = 0; r < R; ++r) {
							float2 p = unpack2(pq[r]);
#pragma unroll
							for (int j = 0; j < PY; ++j)
								p.x = fmaf(unpack2(ph[j]).x, win[LH + r - j], p.x);
							pq[r] = pack2(p.x, p.y);
						}
					}
				}
			};
			if (all_lo) rows(std::true_type{}); else rows(std::false_type{});
#pragma unroll
			for (int r = 0; r < R; ++r) {
				const float2 p = unpack2(pq[r]);
				kahan_add(s[r], c[r], p.x + p.y);
			}
		}

		// 4. S = noise + all terms outside the unknown in-tile part
		if (grp == 1) {
#pragma unroll
			for (int q = 0; q < R / 4; ++q)
				reinterpret_cast<float4*>(comb)[q * GROUP + lt] =
				    make_float4(s[4 * q] - c[4 * q], s[4 * q + 1] - c[4 * q + 1],
				                s[4 * q + 2] - c[4 * q + 2], s[4 * q + 3] - c[4 * q + 3]);
		}
		bar_sync(BAR_COMP, NCOMP);
		if (grp == 0) {
#pragma unroll
			for (int q = 0; q < R / 4; ++q) {
				const float4 v = reinterpret_cast<const float4*>(comb)[q * GROUP + lt];
				const float g1[4] = {v.x, v.y, v.z, v.w};
				float o[4];
#pragma unroll
				for (int e = 0; e < 4; ++e) {
					const int r = 4 * q + e;
					const bool valid = gx < tk.nx && y0 + yl0 + r < tk.ny;
					o[e] = valid ? (s[r] + (g1[e] - c[r])) : 0.0f;
				}
				reinterpret_cast<float4*>(ss + xl * SW + SPAD + yl0)[q] =
				    make_float4(o[0], o[1], o[2], o[3]);
			}
		}
		bar_sync(BAR_COMP, NCOMP);

		//    zeta = H * S over the quarter plane of the tile, in work units
		if (tid < HUNITS) h_unit(ss, sh_h, hu, tid, part);

		// 5. sum each output's unit partials (Kahan, in dx order), store the
		//    solved slice; the halo warp publishes it
		bar_sync(BAR_COMP, NCOMP);
		{
			// this thread's outputs: row ox, columns oy0 .. oy0+3
			const int ox = tid / (2 * STRIPS);
			const int ostrip = (tid / 2) % STRIPS;
			const int oy0 = ostrip * R + (tid % 2) * 4;
			const int opart = (ostrip == 0 || ostrip == 3 ? 0 : HPAIR) + ox;
			const int oslot = (ostrip >= 2 ? 0 : R) + (tid % 2) * 4;
			const int ogx = x0 + ox;
			float a[4], ac[4];
#pragma unroll
			for (int e = 0; e < 4; ++e) { a[e] = 0.0f; ac[e] = 0.0f; }
			const int nch = ox / HCH + 1;
			for (int ch = 0; ch < nch; ++ch) {
				const float4 v = *reinterpret_cast<const float4*>(part + (opart + h_start(ch) - HCH * ch) * PS + oslot);
				kahan_add(a[0], ac[0], v.x);
				kahan_add(a[1], ac[1], v.y);
				kahan_add(a[2], ac[2], v.z);
				kahan_add(a[3], ac[3], v.w);
			}
#pragma unroll
			for (int e = 0; e < 4; ++e) a[e] -= ac[e];
			const float4 z4 = make_float4(a[0], a[1], a[2], a[3]);
			*reinterpret_cast<float4*>(cur + (hx + ox) * W + LH + oy0) = z4;
			bar_sync(BAR_COMP, NCOMP);  // slice t in the ring for every compute thread
			// (released before this slice's global stores: it waits for none)
			if (tid == 0) st_release_cta(&sh->done, t + 1);
			float* zo = zt + (long long)ogx * tk.ny + y0 + oy0;
			if (ogx < tk.nx && vec) {
				if (y0 + oy0 < tk.ny) *reinterpret_cast<float4*>(zo) = z4;
			} else if (ogx < tk.nx) {
#pragma unroll
				for (int e = 0; e < 4; ++e)
					if (y0 + oy0 + e < tk.ny) zo[e] = a[e];
			}
		}
		// the barrier's previous round is over once the publication warp has
		// left it (it waits for nothing but these barriers)
		for (long long it = 0; *((volatile int*)&sh->published) < t + 1 - PUB_BARS; ++it)
			if (it == 64ll * kSpinLimit) {
				atomicExch(err, DEV_TIMEOUT);
				break;
			}
		__syncwarp();
		bar_arrive(BAR_PUB + t % PUB_BARS, NTHREADS);
	}
}

// A tile's coefficients, H, zeroed ring and history into shared memory.  (Each kernel
// has its own copy, whose registers are allocated with the kernel's.)
template <bool BY_TASK>
__device__ __noinline__ void stage_tile(const Task& tk, int bx, int by, const Layout& L,
                                        float* smem, unsigned char* s_lo) {
	const int tid = threadIdx.x;
	const int pt = tk.pt, px = tk.px, py = tk.py, pyp = L.pyp;
	const int x0 = bx * TX, y0 = by * TY;
	const long long sst = (long long)tk.nx * tk.ny;
	float* ring = smem;
	float* sphi = ring + L.slots * L.slot_sz;
	float* sh_h = sphi + 2 * L.taps;
	float* ss = sh_h + TX * HS;
	// coefficient rows padded with zeros, H, the ring and S pads zero
	for (int q = tid; q < L.taps; q += NTHREADS) {
		const int j = q % pyp, ki = q / pyp;
		sphi[2 * q] = j < py ? tk.phi[ki * py + j] : 0.0f;
		sphi[2 * q + 1] = j < py ? tk.phi_lo[ki * py + j] : 0.0f;
	}
	// rows whose lo parts are all zero skip their second FMA chain
	for (int ki = tid; ki < pt * px; ki += NTHREADS) {
		bool nz = false;
		for (int j = 0; j < py; ++j) nz = nz || tk.phi_lo[ki * py + j] != 0.0f;
		s_lo[ki] = nz ? 1 : 0;
	}
	for (int q = tid; q < TX * TY; q += NTHREADS) sh_h[(q / TY) * HS + q % TY] = tk.h[q];
	for (int q = tid; q < L.slots * L.slot_sz; q += NTHREADS) ring[q] = 0.0f;
	for (int q = tid; q < TX * SW; q += NTHREADS) ss[q] = 0.0f;
	__syncthreads();
	// history slices (a stream's previous chunk): the whole ring slot, tile
	// and halo, straight from global memory (zero outside the surface)
	for (int tt = max(0, tk.t0 - pt + 1); tt < tk.t0; ++tt) {
		float* slot = ring + (tt % L.slots) * L.slot_sz;
		const float* zs = tk.zeta + tt * sst;
		for (int q = tid; q < L.slot_sz; q += NTHREADS) {
			const int x = x0 - L.hx + q / W, y = y0 - LH + q % W;
			if (x >= 0 && x < tk.nx && y >= 0 && y < tk.ny)
				slot[q] = __ldcg(zs + (long long)x * tk.ny + y);
		}
	}
}

// Tile k of a grid of a x b tiles by anti-diagonals: a tile's neighbours x - 1, y - 1
// and both come before it.
__device__ int2 diagonal_tile(int k, int a, int b) {
	const int m = min(a, b), head = m * (m - 1) / 2;  // tiles on diagonals shorter than m
	const bool tail = k >= a * b - head;              // the last ones mirror the first
	if (tail) k = a * b - 1 - k;
	int2 t;
	if (k < head) {
		int d = int((sqrtf(8.0f * float(k) + 1.0f) - 1.0f) * 0.5f);
		while (d * (d + 1) / 2 > k) --d;
		while ((d + 1) * (d + 2) / 2 <= k) ++d;
		t.x = k - d * (d + 1) / 2;
		t.y = d - t.x;
	} else {
		const int q = k - head, d = m - 1 + q / m;
		t.x = a <= b ? q % m : d - q % m;
		t.y = d - t.x;
	}
	return tail ? make_int2(a - 1 - t.x, b - 1 - t.y) : t;
}

// One launch for the whole batch: each ticket's surface selects the
// instantiation for its tap count py (warp-uniform switch).  BY_TASK: lead, pace and
// order of tiles as the task says, else 1, none and by anti-diagonals where they do not
// all run at once (a kernel of its own: with the choice in one, 512 x 256 x 256 of order
// 10^3, which needs none of it, took 1 to 2 % longer).
template <bool BY_TASK>
__global__ void __launch_bounds__(NTHREADS, 3)
ar32c_kernel(const Task* __restrict__ tasks, int ntasks, int total_tickets,
             int* __restrict__ ticket_counter, int* __restrict__ err) {
	extern __shared__ __align__(16) float smem[];
	__shared__ int s_ticket;
	__shared__ Progress sh;
	__shared__ unsigned char s_lo[kMaxTapRows];  // per (k, i) tap row: lo part present
	const int tid = threadIdx.x;
	for (;;) {
		if (tid == 0)
			s_ticket = *((volatile int*)err) == DEV_OK ? atomicAdd(ticket_counter, 1) : total_tickets;
		__syncthreads();
		const int ticket = s_ticket;
		__syncthreads();
		if (ticket >= total_tickets) return;
		// locate the surface owning this ticket
		int lo = 0, hi = ntasks - 1;
		while (lo < hi) {
			const int mid = (lo + hi + 1) / 2;
			if (tasks[mid].ticket_base <= ticket) lo = mid; else hi = mid - 1;
		}
		const Task tk = tasks[lo];
		const int local = ticket - tk.ticket_base;
		int bx = local / tk.tiles_y, by = local % tk.tiles_y;
		if (BY_TASK ? tk.diagonal : total_tickets > int(gridDim.x)) {
			const int2 tile = diagonal_tile(local, tk.tiles_x, tk.tiles_y);
			bx = tile.x;
			by = tile.y;
		}
		if (bx < tk.given_tx) {
			// a given tile (the band above an x-strip, holding the upper strip's
			// finished values): published as complete for every slice at once
			if (tid == 0) st_release(tk.flags + bx * tk.tiles_y + by, tk.nt);
			continue;
		}
		const Layout L = tile_layout(tk.pt, tk.px, tk.py, BY_TASK ? tk.lead : 1);
		stage_tile<BY_TASK>(tk, bx, by, L, smem, s_lo);
		if (tid == 0) {
			sh.done = tk.t0;
			sh.published = tk.t0;
		}
		__syncthreads();
		if (tid >= NCOMP) {
			halo_warp<BY_TASK>(tk, bx, by, L, smem, &sh, err);
		} else {
			switch (tk.py) {
#define ARMA_PY_CASE(N) case N: compute_tile<N>(tk, bx, by, L, smem, s_lo, &sh, err); break;
				ARMA_PY_CASE(1) ARMA_PY_CASE(2) ARMA_PY_CASE(3) ARMA_PY_CASE(4) ARMA_PY_CASE(5)
				ARMA_PY_CASE(6) ARMA_PY_CASE(7) ARMA_PY_CASE(8) ARMA_PY_CASE(9) ARMA_PY_CASE(10)
				ARMA_PY_CASE(11) ARMA_PY_CASE(12) ARMA_PY_CASE(13)
#undef ARMA_PY_CASE
				default: break;
			}
		}
		__syncthreads();
	}
}

constexpr size_t kStaticSmem = 256;  // no less than ar32c_kernel has: ticket, progress, lo rows

size_t smem_bytes(int pt, int px, int py, int lead) {
	const Layout l = tile_layout(pt, px, py, lead);
	return sizeof(float) * (size_t(l.slots) * l.slot_sz + 2 * size_t(l.taps) + TX * HS + TX * SW +
	                        std::max(GROUP * R, HUNITS * PS));
}

// What decides how many CTAs share an SM.
struct Load32 {
	double tiles = 0, work = 0, spread = 0;  // tiles, their slices' cost, their surfaces' chains
	double chain = 0;                        // the longest chain of slices, by cost
	int taps = 0;                            // of its surface
	// a surface's wavefront needs about nt + tiles_x + tiles_y slice steps, each
	// proportional to its taps and what H and the sums cost (as much as 160 taps)
	static double chain_of(const Ar32Surface& s) {
		return double(s.nt - s.t0 + s.tiles_x + s.tiles_y) * (s.pt * s.px * s.py + 160);
	}
	void add(const Ar32Surface& s) {
		const double n = double(s.tiles_x - s.given_tx) * s.tiles_y, c = chain_of(s);
		tiles += n;
		work += n * (s.nt - s.t0) * (s.pt * s.px * s.py + 160);
		spread += n * c;
		if (c > chain) taps = s.pt * s.px * s.py;
		chain = std::max(chain, c);
	}
	double at_work() const { return work / chain; }
	bool alike() const { return spread >= 0.9 * tiles * chain; }
};

// CTAs per SM for a launch, of `most` that fit.  Of all tiles, work / chain are at
// work at once if none waits for an SM.  CTAs that share an SM slow each other's
// chains: in a batch of different surfaces, below about one such tile per SM the
// longest chain is left an SM to itself, and below 2.4 it shares with one other.
// Measured with one, two and three per SM (ms): 0.9 tiles per SM 3.9 / 5.4 / 5.3;
// 1.3 7.8 / 6.4 / 8.4; 1.7 6.4 / 4.8 / 6.0; 2.0 11.2 / 8.6 / 8.9; 2.8 15.0 / 10.6 /
// 10.1; 3.1 13.3 / 9.5 / 8.8; 4.8 28.4 / 20.2 / 19.0.
// Where all chains are about as long as the longest (one surface, or many alike),
// tiles that find no SM make a second wave as long as the first: the fewest waves,
// each by what its CTAs slow each other (light orders less).  Where few slices leave
// many of the tiles waiting for their first, only those at work count.  200 slices,
// with one, two and three per SM (ms): 196 tiles of 10^3 3.7 / 3.1 / 3.1, 400 5.5 /
// 7.1 / 4.6, 576 7.2 / 7.2 / 10.5, 900 of 4^3 - / 3.1 / 2.7; 60 slices: 400 tiles of
// 10^3 1.7 / 2.0 / 1.7, of 4^3 0.68 / 0.68 / 0.77.
// More than `with_lead` CTAs only fit without the halo a slice ahead (launch_ar32c): of
// tiles alike, where they then all run at once.
int ctas_per_sm(const Load32& l, int sms, int most, int with_lead) {
	const double at_work = l.at_work();
	if (!l.alike()) return at_work < 1.1 * sms ? 1 : at_work < 2.4 * sms ? std::min(2, most) : most;
	const bool heavy = l.taps >= kHeavyTaps;
	const double slowed[] = {1.0, heavy ? 1.6 : 1.45, heavy ? 2.45 : 1.9};
	const bool few = at_work < (heavy ? 0.5 : 0.75) * l.tiles;  // at work at once
	int best = 1;
	double least = HUGE_VAL;
	for (int n = 1; n <= std::min(most, 3); ++n) {
		if (n > with_lead && l.tiles > n * sms) continue;
		const double waves = few ? std::max(1.0, at_work / (n * sms)) : std::ceil(l.tiles / (n * sms));
		const double time = slowed[n - 1] * waves;
		if (time < least) {
			least = time;
			best = n;
		}
	}
	return best;
}

// How a launch's tiles share the device, by task.
//
// Tiles of many taps keep pace with the tiles below them where several run on an SM
// and all run at once: one that is far ahead takes the SM from the tiles that the
// rest of the surface waits for (200 slices of 10^3, 400 tiles on 444 CTAs: 4.6 to 7.3
// ms, 4.7 keeping pace).  Tiles that wait for a CTA are the sooner served the sooner
// others end, and tiles of few taps lose more than they gain (1^3, 400 tiles: 1.6 /
// 2.2 ms).
//
// Tiles that do not all run at once are handed out by anti-diagonals, a front across
// the surface.  Row by row they are a band of rows end to end, of which only the
// stretch that the slices span is at work (60 x 1024 x 2048 of order 4^3 5.0 / 3.1 ms,
// 20 x 96 x 1920 of 8^3 0.86 / 0.52; the batch of 256 surfaces 48.3 / 48.3).  Where that
// is most of it, tiles of many taps crowd each other out less row by row (200 x 384 x
// 768 of 10^3 6.9 / 7.2).
void share_device(Task& t, const Load32& l, int total, int grid, int sms) {
	t.pace = t.pt * t.px * t.py >= kHeavyTaps && total <= grid && total > sms;
	t.diagonal = total > grid &&
	             !(l.alike() && l.taps >= kHeavyTaps && l.at_work() >= 0.75 * l.tiles);
}

}  // namespace

void launch_ar32c_starved(Ctx* c) {
	const size_t words = 2 * size_t(TX) * 2 * TY + 2 * 2 + size_t(TX) * TY;
	auto* zeta = static_cast<float*>(scratch_take(c, sizeof(float) * words));
	int* flags = static_cast<int*>(scratch_take(c, sizeof(int) * 3));
	ARMA_CUDA_TRY(cudaMemsetAsync(zeta, 0, sizeof(float) * words, c->stream));
	Task t{};
	t.nt = 2; t.nx = TX; t.ny = 2 * TY;
	t.pt = t.px = 1; t.py = 2;
	t.lead = 1;
	t.tiles_x = 1; t.tiles_y = 2;
	t.polls = kStarvedPolls;
	t.zeta = zeta;
	t.phi = zeta + 2 * size_t(TX) * 2 * TY;
	t.phi_lo = t.phi + 2;
	t.h = t.phi_lo + 2;
	t.flags = flags;
	auto* d_task = static_cast<Task*>(scratch_take(c, sizeof(Task)));
	const int start[3] = {0, 0, 1};  // nothing published; the next ticket: the second tile
	ARMA_CUDA_TRY(copy_async(c, d_task, &t, sizeof(t), cudaMemcpyHostToDevice, c->stream));
	ARMA_CUDA_TRY(copy_async(c, flags, start, sizeof(start), cudaMemcpyHostToDevice, c->stream));
	const size_t smem = smem_bytes(t.pt, t.px, t.py, t.lead);
	allow_smem(ar32c_kernel<false>, smem, kStaticSmem);
	ProfScope prof_(c, "ar32c");
	ar32c_kernel<false><<<1, NTHREADS, smem, c->stream>>>(d_task, 1, 2, flags + 2, c->d_err);
	ARMA_CUDA_TRY(cudaGetLastError());
	c->launches += 1;
}

int ar32c_tile_x() { return TX; }
int ar32c_tile_y() { return TY; }
int ar32c_max_tap_rows() { return kMaxTapRows; }

void launch_ar32c(Ctx* c, const std::vector<Ar32Surface>& surfaces, int tx, int ty, int) {
	ARMA_REQUIRE(tx == TX && ty == TY, ARMA_EINVAL, "unsupported AR tile shape");
	std::vector<int> order(surfaces.size());
	size_t most_bytes[2] = {0, 0};  // of a tile, by its lead
	for (size_t k = 0; k < surfaces.size(); ++k) {
		const Ar32Surface& s = surfaces[k];
		ARMA_REQUIRE(s.px <= TX + 1 && s.py <= MAXO && s.pt >= 1 && s.px >= 1 && s.py >= 1 &&
		                 s.pt * s.px <= kMaxTapRows,
		             ARMA_ENOTSUP, "AR order not supported by the FP32 tile kernel");
		order[k] = int(k);
		for (int lead : {0, 1})
			most_bytes[lead] = std::max(most_bytes[lead], smem_bytes(s.pt, s.px, s.py, lead));
	}
	// longest dependency chains first
	std::sort(order.begin(), order.end(), [&](int a, int b) {
		return Load32::chain_of(surfaces[a]) > Load32::chain_of(surfaces[b]);
	});
	size_t nflags = 0;
	Load32 load;
	for (const auto& s : surfaces) {
		nflags += size_t(s.tiles_x) * s.tiles_y;
		load.add(s);
	}
	int* flags = static_cast<int*>(scratch_take(c, sizeof(int) * nflags));
	ARMA_CUDA_TRY(cudaMemsetAsync(flags, 0, sizeof(int) * nflags, c->stream));
	std::vector<Task> tasks;
	int total = 0;
	size_t foff = 0;
	for (int k : order) {
		const Ar32Surface& s = surfaces[k];
		Task t;
		t.nt = s.nt; t.nx = s.nx; t.ny = s.ny;
		t.pt = s.pt; t.px = s.px; t.py = s.py;
		t.t0 = s.t0;
		t.given_tx = s.given_tx;
		t.tiles_x = s.tiles_x; t.tiles_y = s.tiles_y;
		t.ticket_base = total;
		t.polls = kSpinLimit;
		t.zeta = s.zeta; t.phi = s.phi; t.phi_lo = s.phi_lo; t.h = s.h;
		t.flags = flags + foff;
		foff += size_t(s.tiles_x) * s.tiles_y;
		total += s.tiles_x * s.tiles_y;
		tasks.push_back(t);
	}
	auto fit = [&](size_t bytes) {  // CTAs on an SM
		allow_smem(ar32c_kernel<false>, bytes, kStaticSmem);
		int n = 0;
		ARMA_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, ar32c_kernel<false>, NTHREADS,
		                                                            bytes));
		return n;
	};
	// The halo a slice ahead takes a slot of the ring, which costs the largest orders
	// a CTA per SM: it is given up where that CTA is wanted (200 x 256 x 512 of order 16
	// x 13 x 9, one CTA with and two without: 6.4 / 5.4 ms; 200 x 320 x 640 of 11 x 10
	// x 10, two and three: 5.9 / 5.1).
	const int with_lead = fit(most_bytes[1]);
	const int most = with_lead < 3 ? fit(most_bytes[0]) : with_lead;
	ARMA_REQUIRE(most > 0, ARMA_EINVAL, "AR tile does not fit in shared memory");
	const int per_sm = c->tuning.ar_ctas_per_sm > 0 ? std::min(most, c->tuning.ar_ctas_per_sm)
	                                                : ctas_per_sm(load, c->num_sms, most, with_lead);
	const size_t smem = most_bytes[per_sm <= with_lead ? 1 : 0];
	const int grid = std::min(total, per_sm * c->num_sms);
	bool by_task = false;
	for (Task& t : tasks) {
		t.lead = smem_bytes(t.pt, t.px, t.py, 1) <= smem;
		share_device(t, load, total, grid, c->num_sms);
		by_task = by_task || !t.lead || t.pace || t.diagonal != (total > grid);
	}
	Task* d_tasks = static_cast<Task*>(scratch_take(c, sizeof(Task) * tasks.size()));
	int* d_ticket = static_cast<int*>(scratch_take(c, sizeof(int)));
	ARMA_CUDA_TRY(copy_async(c, d_tasks, tasks.data(), sizeof(Task) * tasks.size(),
	                              cudaMemcpyHostToDevice, c->stream));
	ARMA_CUDA_TRY(cudaMemsetAsync(d_ticket, 0, sizeof(int), c->stream));
	ProfScope prof_(c, "ar32c");
	auto kernel = ar32c_kernel<false>;
	if (by_task) {
		kernel = ar32c_kernel<true>;
		allow_smem(kernel, smem, kStaticSmem);
	}
	kernel<<<grid, NTHREADS, smem, c->stream>>>(d_tasks, int(tasks.size()), total, d_ticket, c->d_err);
	ARMA_CUDA_TRY(cudaGetLastError());
	c->launches += 1;
}

}  // namespace armab

// ---------------------------------------------------------------------------
// Allocation-free entry point.
//
// Some callers cannot allocate device memory at the point where they filter a
// surface: code that runs inside another framework's memory pool and must not
// make stray cudaMalloc calls, latency-bound serving loops that forbid
// allocation (and its implicit synchronisation) on the request path, and
// plugins loaded into processes whose allocator owns the whole device.  This
// entry point runs the same FP32 filter kernel on one surface with every
// piece of scratch it needs (the tile task, the ticket counter, the error
// word, the per-tile publication counters and the hi/lo coefficient and
// intra-slice-response tables) in one file-scope __device__ array of
// kStaticScratchBytes (64 KiB), which every GPU that loads this library holds
// until the process exits.
//
//   * Limits: at most kStaticMaxTiles (8192) tiles of 16 x 32 points per time
//     slice and at most kStaticMaxTaps (2048) AR coefficients; larger
//     requests are rejected with ARMA_EINVAL.  Orders follow the FP32 filter's
//     own limits (at most 16 per axis, px <= 17, py <= 13, pt * px <= 221)
//     and answer ARMA_ENOTSUP beyond them, as arma_ar_filter does.
//   * The coefficient tables are the ones the context path builds
//     (ar32_coefficients), so the result is bit-identical to
//     arma_ar_filter(..., ARMA_FP32C, ...) on the same input.
//   * The first call on a device looks up the array's device address with
//     cudaGetSymbolAddress (once per device, under a lock).
//   * Every call reads the device error word back and synchronises the
//     stream before it returns, and stages its tables from host stack
//     memory, so it cannot run under stream capture: a capturing stream is
//     refused with ARMA_EINVAL.
//   * Every call reuses the same array and leaves the last call's contents in
//     it; each call clears the counters it relies on.  Calls whose work
//     overlaps on the GPU (other streams or threads) race on the array and
//     must be serialised by the caller.
//   * It calls no cudaMalloc, cudaFree or allocating library routine.
namespace armab {
namespace {

constexpr size_t kStaticScratchBytes = 64 * 1024;
constexpr int kStaticMaxTiles = 8192;
constexpr int kStaticMaxTaps = 2048;
// byte offsets inside the array; the coefficient block is hi[P], lo[P], H[TX*TY]
constexpr size_t kOffTask = 0;
constexpr size_t kOffTicket = 256;
constexpr size_t kOffErr = 260;
constexpr size_t kOffFlags = 512;
constexpr size_t kOffCoef = kOffFlags + sizeof(int) * kStaticMaxTiles;
constexpr size_t kMaxCoefFloats = 2 * size_t(kStaticMaxTaps) + size_t(TX) * TY;
constexpr size_t kStaticEnd = kOffCoef + sizeof(float) * kMaxCoefFloats;
static_assert(kStaticEnd <= kStaticScratchBytes, "static scratch layout overflows");
static_assert(sizeof(Task) <= kOffTicket, "task record overflows its slot");

static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];

constexpr int kMaxDevices = 64;
std::mutex g_static_lock;
unsigned char* g_static_addr[kMaxDevices] = {nullptr};

// The array's device address on the current device (looked up once per
// device); nullptr when the lookup fails.
unsigned char* static_scratch(int dev) {
	std::lock_guard<std::mutex> lk(g_static_lock);
	if (!g_static_addr[dev]) {
		void* p = nullptr;
		if (cudaGetSymbolAddress(&p, g_static_scratch) != cudaSuccess) return nullptr;
		g_static_addr[dev] = static_cast<unsigned char*>(p);
	}
	return g_static_addr[dev];
}

}  // namespace
}  // namespace armab

extern "C" int arma_ar_filter_fp32c_noalloc(void* stream, const double* phi, const int order[3],
                                            const int shape[3], float* d_zeta) {
	using namespace armab;
	// A failed runtime call leaves the runtime's last-error state set; clear it
	// so that neither this call's launch check nor a later one reads it.
	auto fail = [](int code, const char* msg) {
		(void)cudaGetLastError();
		set_error(msg);
		return code;
	};
	(void)cudaGetLastError();
	if (!phi || !order || !shape || !d_zeta) return fail(ARMA_EINVAL, "null argument");
	if (shape[0] <= 0 || shape[1] <= 0 || shape[2] <= 0)
		return fail(ARMA_EINVAL, "Bad \"out_grid\": dimensions must be positive");
	if (order[0] < 1 || order[1] < 1 || order[2] < 1 || order[0] > 16 || order[1] > 16 ||
	    order[2] > 16)
		return fail(ARMA_ENOTSUP, "AR order above 16 per dimension is not supported on the device");
	if (order[1] > TX + 1 || order[2] > MAXO || order[0] * order[1] > kMaxTapRows)
		return fail(ARMA_ENOTSUP, "AR order not supported by the FP32 tile kernel");
	const int P = order[0] * order[1] * order[2];
	if (P > kStaticMaxTaps)
		return fail(ARMA_EINVAL, "allocation-free AR filter: more than 2048 coefficients");
	const int tiles_x = (shape[1] + TX - 1) / TX, tiles_y = (shape[2] + TY - 1) / TY;
	if ((long long)tiles_x * tiles_y > kStaticMaxTiles)
		return fail(ARMA_EINVAL,
		            "allocation-free AR filter: slice needs more than 8192 tiles of 16x32 points");
	cudaStream_t st = static_cast<cudaStream_t>(stream);
	cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
	if (cudaStreamIsCapturing(st, &cap) != cudaSuccess)
		return fail(ARMA_ECUDA, "cudaStreamIsCapturing failed");
	if (cap != cudaStreamCaptureStatusNone)
		return fail(ARMA_EINVAL,
		            "allocation-free AR filter: the stream is capturing (the call synchronises)");
	int dev = 0;
	if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices)
		return fail(ARMA_ECUDA, "cudaGetDevice failed");
	size_t smem = smem_bytes(order[0], order[1], order[2], 1);
	int smem_optin = 0;
	if (cudaDeviceGetAttribute(&smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) !=
	    cudaSuccess)
		return fail(ARMA_ECUDA, "shared-memory limit query failed");
	if (smem + kStaticSmem > size_t(smem_optin))
		return fail(ARMA_ENOTSUP, "AR order needs more shared memory than the device has");
	unsigned char* base = static_scratch(dev);
	if (!base) return fail(ARMA_ECUDA, "cudaGetSymbolAddress of the static scratch failed");
	for (auto kernel : {ar32c_kernel<false>, ar32c_kernel<true>})
		if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
		                         int(kSmemOptin - kStaticSmem)) != cudaSuccess)
			return fail(ARMA_ECUDA, "cudaFuncSetAttribute failed");
	float* d_coef = reinterpret_cast<float*>(base + kOffCoef);
	// the context path's tables (hi/lo split, lo-row selection, H), built into
	// host stack memory: 2P + TX*TY <= kMaxCoefFloats floats
	float cbuf[kMaxCoefFloats];
	const size_t ncoef = ar32_coefficient_count(order);
	ar32_coefficients(phi, order, cbuf);
	Task t;
	t.nt = shape[0]; t.nx = shape[1]; t.ny = shape[2];
	t.pt = order[0]; t.px = order[1]; t.py = order[2];
	t.t0 = 0;
	t.given_tx = 0;
	t.tiles_x = tiles_x; t.tiles_y = tiles_y;
	t.ticket_base = 0;
	t.polls = kSpinLimit;
	t.zeta = d_zeta;
	t.phi = d_coef;
	t.phi_lo = d_coef + P;
	t.h = d_coef + 2 * P;
	t.flags = reinterpret_cast<int*>(base + kOffFlags);
	int* d_ticket = reinterpret_cast<int*>(base + kOffTicket);
	int* d_err = reinterpret_cast<int*>(base + kOffErr);
	const int ntiles = tiles_x * tiles_y;
	const size_t smem0 = smem_bytes(order[0], order[1], order[2], 0);
	int with_lead = 0, most = 0, sms = 0;
	if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&with_lead, ar32c_kernel<false>, NTHREADS,
	                                                  smem) != cudaSuccess ||
	    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&most, ar32c_kernel<false>, NTHREADS, smem0) !=
	        cudaSuccess ||
	    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
		return fail(ARMA_ECUDA, "occupancy query failed");
	if (most <= 0) return fail(ARMA_ENOTSUP, "AR tile does not fit in shared memory");
	Load32 load;
	load.add(Ar32Surface{t.nt, t.nx, t.ny, t.pt, t.px, t.py, d_zeta, t.phi, t.phi_lo, t.h, tiles_x,
	                     tiles_y});
	const int per_sm = ctas_per_sm(load, sms, most, with_lead);
	const int grid = std::min(ntiles, per_sm * sms);
	t.lead = per_sm <= with_lead;
	share_device(t, load, ntiles, grid, sms);
	if (!t.lead) smem = smem0;
	if (cudaMemcpyAsync(base + kOffTask, &t, sizeof(t), cudaMemcpyHostToDevice, st) != cudaSuccess ||
	    cudaMemcpyAsync(d_coef, cbuf, sizeof(float) * ncoef, cudaMemcpyHostToDevice, st) !=
	        cudaSuccess ||
	    cudaMemsetAsync(base + kOffTicket, 0, 8, st) != cudaSuccess ||
	    cudaMemsetAsync(t.flags, 0, sizeof(int) * ntiles, st) != cudaSuccess) {
		(void)cudaStreamSynchronize(st);  // the staged host buffers are on this stack
		return fail(ARMA_ECUDA, "staging the allocation-free AR filter failed");
	}
	const bool by_task = !t.lead || t.pace || t.diagonal != (ntiles > grid);
	auto kernel = by_task ? ar32c_kernel<true> : ar32c_kernel<false>;
	kernel<<<grid, NTHREADS, smem, st>>>(reinterpret_cast<const Task*>(base + kOffTask), 1, ntiles,
	                                     d_ticket, d_err);
	const bool launched = cudaGetLastError() == cudaSuccess;
	int herr = 0;
	const bool copied =
	    cudaMemcpyAsync(&herr, d_err, sizeof(int), cudaMemcpyDeviceToHost, st) == cudaSuccess;
	// wait in every case: the stream still reads this stack's buffers
	const bool synced = cudaStreamSynchronize(st) == cudaSuccess;
	if (!launched) return fail(ARMA_ECUDA, "AR kernel launch failed");
	if (!copied || !synced) return fail(ARMA_ECUDA, "AR kernel failed");
	if (herr == DEV_TIMEOUT)
		return fail(ARMA_ETIMEDOUT, "a bounded device wait gave up (tile dependency not met)");
	if (herr != DEV_OK) return fail(ARMA_ECUDA, "device-side check failed");
	return ARMA_OK;
}
