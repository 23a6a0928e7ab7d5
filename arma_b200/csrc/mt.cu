// dcmt Mersenne Twister word generation on the device.
//
// The dcmt generator (genrand_mt, called by prng::parallel_mt::operator(),
// reference src/parallel_mt.hh:236) is the MT linear recurrence over a ring of
// nn words followed by tempering.  Written as a sequence of raw words
//     x[j] = x[j-n+m] ^ (y >> 1) ^ (y & 1 ? aaa : 0),
//     y    = (x[j-n] & umask) | (x[j-n+1] & lmask),   j >= n,
// with x[0..n-1] the seeded state (sgenrand_mt), output word w is
// temper(x[n+w]).  Every word of a chunk [j0, j0+n-m) depends only on words
// before j0, so one CTA produces n-m words per barrier step with all
// arithmetic in 32-bit integers; sets with nn = 2 mm run one warp per segment
// with no barrier (mt_generate_half_kernel).
//
// Long streams are cut into segments of J = 2^v words (segment_log2) generated
// by separate CTAs or warps.  The window of nn raw words at the start of segment
// k is obtained by jumping: with g(t) = t^(J 2^l) mod phi(t) (phi the
// characteristic polynomial, mt_jump.cc), the window D positions ahead is the
// XOR of the windows of the raw sequence at the set bits of g.  Segment starts
// are built as a binary tree: level l turns every known start k*2^(l+1) into
// k*2^(l+1) + 2^l.  All of it is bit-identical to the sequential generator.
#include <algorithm>
#include <cstring>
#include <map>
#include <mutex>
#include <vector>

#include "internal.h"

namespace armab {

// Defined in mt_jump.cc: the coefficients of t^(2^e) mod phi, bit i of word i /
// 32; false when no polynomial of degree 32 nn - rr is found that the sequence obeys.
bool mt_jump_bits(const arma_mt_params& prm, int e, std::vector<uint32_t>* bits);

namespace {

constexpr int kRingBits = 12;
constexpr int kRing = 1 << kRingBits;  // ring of raw words, >= nn + (nn-mm)
constexpr int kLevels = 16;            // at most 2^16 segments
constexpr int kMinLog2Seg = 16;        // shortest segment of the rule below
// more segments per SM than this are generated by a warp each
constexpr size_t kWarpSegments = 6;
constexpr int kJumpThreads = 384;

struct SegJob {
	arma_mt_params p;
	uint32_t seed;
	const uint32_t* state;     // window of nn raw words, or null: seed it
	unsigned long long first;  // output index of the segment's first word
	unsigned long long count;  // words in the segment
	unsigned long long offset; // words before `offset` are not stored
	uint32_t* out;             // out[w - offset] for output index w
};

struct JumpJob {
	arma_mt_params p;
	const uint32_t* src;  // window at position a
	uint32_t* dst;        // window at position a + D (zero when parts > 1)
	const uint32_t* bits; // t^D mod phi, bit i of word i / 32
};

__device__ __forceinline__ uint32_t temper(uint32_t y, const arma_mt_params& p) {
	y ^= y >> p.shift0;
	y ^= (y << p.shiftB) & p.maskB;
	y ^= (y << p.shiftC) & p.maskC;
	y ^= y >> p.shift1;
	return y;
}

__device__ __forceinline__ void seed_state(uint32_t* dst, uint32_t seed, const arma_mt_params& p) {
	// sgenrand_mt: Knuth's 1812433253 initialisation masked by wmask.
	uint32_t s = seed;
	for (int k = 0; k < p.nn; ++k) {
		dst[k] = s & p.wmask;
		s = 1812433253u * (s ^ (s >> 30)) + uint32_t(k + 1);
	}
}

// The block has one thread per word of a chunk of n - m words, rounded up
// to whole warps (up to kGenMaxThreads); longer chunks give each thread W =
// ceil((n - m) / blockDim) words (n - m <= kMaxOwn * kGenMaxThreads covers
// every Mersenne exponent up to 44497 several times over).
constexpr int kGenMaxThreads = 1024;
constexpr int kMaxOwn = 4;

template <int W>
__global__ void __launch_bounds__(kGenMaxThreads)
mt_generate_kernel(const SegJob* __restrict__ jobs) {
	__shared__ uint32_t ring[kRing];
	const SegJob& jb = jobs[blockIdx.x];
	const arma_mt_params p = jb.p;
	const int n = p.nn, m = p.mm;
	const int chunk = n - m;
	const long long count = (long long)jb.count;
	const long long shift = (long long)jb.first - (long long)jb.offset;  // out index - word
	uint32_t* const out = jb.out;
	if (jb.state) {
		for (int k = threadIdx.x; k < n; k += blockDim.x) ring[k] = jb.state[k];
	} else if (threadIdx.x == 0) {
		seed_state(ring, jb.seed, p);
	}
	__syncthreads();
	const uint32_t mask = kRing - 1;
	// Thread t owns words t + i B (B = blockDim, i < W, those < n - m) of every
	// chunk: segment word w = s (n-m) + t + i B at step s, raw word r = n + w
	// at ring position r & mask (positions run modulo 2^32, a multiple of the
	// ring size), so every index is a running register sum.  Each step emits
	// the chunk computed by the step before and computes the next one: raw
	// r + n - m reads raw r (this thread's own word) and raw r - m, r - m + 1,
	// all written in earlier steps.
	auto next_word = [&](uint32_t r) {  // raw word r from raw r - n, r - n + 1, r - n + m
		const uint32_t y = (ring[(r - n) & mask] & p.umask) | (ring[(r - n + 1) & mask] & p.lmask);
		return ring[(r - n + m) & mask] ^ (y >> 1) ^ ((y & 1u) ? p.aaa : 0u);
	};
	uint32_t r[W];
	long long o[W], rem[W];
	bool owner[W];
#pragma unroll
	for (int i = 0; i < W; ++i) {
		const int t = threadIdx.x + i * int(blockDim.x);
		owner[i] = t < chunk;
		r[i] = uint32_t(n + t);  // raw position of this word
		o[i] = shift + t;        // its output index
		rem[i] = count - t;      // words from it to the segment's end
		if (owner[i] && rem[i] > 0) ring[r[i] & mask] = next_word(r[i]);
	}
	__syncthreads();
	const long long steps = (count + chunk - 1) / chunk;
	for (long long st = 0; st < steps; ++st) {
#pragma unroll
		for (int i = 0; i < W; ++i) {
			if (owner[i]) {
				if (rem[i] > 0 && o[i] >= 0) out[o[i]] = temper(ring[r[i] & mask], p);
				if (rem[i] > chunk) ring[(r[i] + chunk) & mask] = next_word(r[i] + chunk);
				r[i] += chunk;
				o[i] += chunk;
				rem[i] -= chunk;
			}
		}
		__syncthreads();
	}
}

// Sets with nn = 2 mm (every committed set of period 2^19937 - 1): with the
// chunk n - m = m, output word w = m s + t (step s, slot t < m) is
//     x[n + w] = x[n + w - m] ^ f(x[w], x[w + 1]),
// where x[n + w - m] is slot t of step s-1, x[w] slot t of step s-2 and
// x[w + 1] slot t+1 of step s-2 (slot 0 of step s-1 when t = m-1): every
// word needs only its own slot's last two values and the next slot's.  One
// warp runs one segment with no barrier: lane l holds slots t = 32 q + l
// (q < kHalfQ) of the last two steps in registers, takes the next slot's
// values by shuffles, and stores each q's 32 words coalesced.  The state
// window (raw words 0 .. n-1) is steps -2 and -1.
constexpr int kHalfQ = 10;     // slots per lane: mm <= 320
constexpr int kHalfWarps = 4;  // warps (segments) per CTA
constexpr int kHalfMaxN = 2 * 32 * kHalfQ;

// (mm > 2: half_four reads up to x[t + 2] of a step before it exists)
__host__ __device__ inline bool half_set(const arma_mt_params& p) {
	return p.nn == 2 * p.mm && p.mm > 2 && p.mm <= 32 * kHalfQ;
}

// One step of the warp generator: slots of step s from those of steps s-2 (a)
// and s-1 (b); b0 = slot 0 of step s-1.  M > 0: the compile-time mm (slot
// checks resolved at compile time); M = 0: mm = m at run time.
template <int M>
__device__ __forceinline__ void half_step(const uint32_t* a, const uint32_t* b, uint32_t* nb,
                                          uint32_t b0, int m, int lane, const arma_mt_params& p) {
	const int mm = M > 0 ? M : m;
#pragma unroll
	for (int q = 0; q < kHalfQ; ++q) {
		if (M > 0 && 32 * q >= M) break;
		const int t = 32 * q + lane;
		const uint32_t down = __shfl_down_sync(0xffffffffu, a[q], 1);
		const uint32_t wrap = __shfl_sync(0xffffffffu, q + 1 < kHalfQ ? a[q + 1] : 0u, 0);
		uint32_t a1 = lane < 31 ? down : wrap;
		if ((M == 0 || 32 * q + 31 >= M - 1) && t == mm - 1) a1 = b0;
		const uint32_t y = (a[q] & p.umask) | (a1 & p.lmask);
		nb[q] = b[q] ^ (y >> 1) ^ ((y & 1u) ? p.aaa : 0u);
	}
}

template <int M>
__global__ void __launch_bounds__(32 * kHalfWarps)
mt_generate_half_kernel(const SegJob* __restrict__ jobs, int njobs) {
	__shared__ uint32_t seeded[kHalfWarps][kHalfMaxN];
	const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
	const int g = blockIdx.x * kHalfWarps + wl;
	if (g >= njobs) return;
	const SegJob& jb = jobs[g];
	const arma_mt_params p = jb.p;
	const int m = M > 0 ? M : p.mm;
	const uint32_t* st = jb.state;
	if (!st) {
		if (lane == 0) seed_state(seeded[wl], jb.seed, p);
		__syncwarp();
		st = seeded[wl];
	}
	uint32_t a[kHalfQ], b[kHalfQ];  // slots of steps s-2 and s-1
#pragma unroll
	for (int q = 0; q < kHalfQ; ++q) {
		const int t = 32 * q + lane;
		a[q] = t < m ? st[t] : 0u;
		b[q] = t < m ? st[m + t] : 0u;
	}
	// segment words w < count (<= 2^30) go to out[first - offset + w] when that
	// index is >= 0: base = out + max(first - offset, 0), index w - wmin
	const int count = int(jb.count);
	const long long shift = (long long)jb.first - (long long)jb.offset;
	const int wmin = shift < 0 ? int(-shift) : 0;
	uint32_t* const base = jb.out + (shift > 0 ? shift : 0);
	int w0 = 0;
	if (wmin == 0) {
		// whole steps: every slot < m is stored
		for (; w0 + m <= count; w0 += m) {
			const uint32_t b0 = __shfl_sync(0xffffffffu, b[0], 0);
			uint32_t nb[kHalfQ];
			half_step<M>(a, b, nb, b0, m, lane, p);
			uint32_t* dst = base + w0 + lane;
#pragma unroll
			for (int q = 0; q < kHalfQ; ++q) {
				if (M > 0 && 32 * q >= M) break;
				if ((M > 0 && 32 * q + 32 <= M) || 32 * q + lane < m) dst[32 * q] = temper(nb[q], p);
				a[q] = b[q];
				b[q] = nb[q];
			}
		}
	}
	// the rest: skipped words before the offset, the last partial step
	for (; w0 < count; w0 += m) {
		const uint32_t b0 = __shfl_sync(0xffffffffu, b[0], 0);
		uint32_t nb[kHalfQ];
		half_step<M>(a, b, nb, b0, m, lane, p);
#pragma unroll
		for (int q = 0; q < kHalfQ; ++q) {
			const int t = 32 * q + lane;
			const int w = w0 + t;
			if (t < m && w < count && w >= wmin) base[w - wmin] = temper(nb[q], p);
			a[q] = b[q];
			b[q] = nb[q];
		}
	}
}

// A set's recurrence and tempering constants held in registers (opaque to the
// compiler, which otherwise loads them again in every step).
__device__ __forceinline__ arma_mt_params in_registers(arma_mt_params p) {
	asm volatile("" : "+r"(p.aaa), "+r"(p.umask), "+r"(p.lmask), "+r"(p.maskB), "+r"(p.maskC));
	asm volatile("" : "+r"(p.shift0), "+r"(p.shift1), "+r"(p.shiftB), "+r"(p.shiftC));
	asm volatile("" : "+r"(p.nn), "+r"(p.mm), "+r"(p.rr));
	return p;
}

__device__ __forceinline__ uint32_t twist(uint32_t u, uint32_t v, const arma_mt_params& p) {
	const uint32_t y = (u & p.umask) | (v & p.lmask);
	return (y >> 1) ^ ((y & 1u) ? p.aaa : 0u);
}

// The same sets with one CTA per segment, a thread per slot, for few segments.
// Words are a CTA's time here, not the GPU's, so a barrier is paid once per four
// steps: from the window of the last two steps (x[0 .. 2 mm)) thread t computes
// its own slot's next four words C, D, E, F, and its right neighbour's C and D,
// which E and F need, once more from the window.  The neighbours of the last two
// slots are the first words of the next step (x[2 mm], x[2 mm + 1]).
__device__ __forceinline__ void half_four(const uint32_t* x, int t, int mm,
                                          const arma_mt_params& p, uint32_t (&w)[4]) {
	const uint32_t a0 = x[t], a1 = x[t + 1], a2 = x[t + 2], b0 = x[mm + t];
	uint32_t b1, b2;
	if (t + 2 < mm) {
		b1 = x[mm + t + 1];
		b2 = x[mm + t + 2];
	} else {
		const uint32_t n0 = x[mm] ^ twist(x[0], x[1], p), n1 = x[mm + 1] ^ twist(x[1], x[2], p);
		b1 = t + 1 < mm ? x[mm + t + 1] : n0;
		b2 = t + 1 < mm ? n0 : n1;
	}
	w[0] = b0 ^ twist(a0, a1, p);
	const uint32_t c1 = b1 ^ twist(a1, a2, p);
	w[1] = w[0] ^ twist(b0, b1, p);
	const uint32_t d1 = c1 ^ twist(b1, b2, p);
	w[2] = w[1] ^ twist(w[0], c1, p);
	w[3] = w[2] ^ twist(w[1], d1, p);
}

constexpr int kFourThreads = 32 * kHalfQ;

__global__ void __launch_bounds__(kFourThreads)
mt_generate_four_kernel(const SegJob* __restrict__ jobs) {
	__shared__ uint32_t win[2][kHalfMaxN + 2];  // (the last two slots read past their step)
	const SegJob& jb = jobs[blockIdx.x];
	const arma_mt_params p = in_registers(jb.p);
	const int mm = p.mm, t = threadIdx.x;
	if (jb.state) {
		for (int k = t; k < p.nn; k += kFourThreads) win[0][k] = jb.state[k];
	} else if (t == 0) {
		seed_state(win[0], jb.seed, p);
	}
	__syncthreads();
	// segment word w < count (<= 2^30) goes to out[first - offset + w] when that
	// index is >= 0
	const int count = int(jb.count);
	const long long shift = (long long)jb.first - (long long)jb.offset;
	const int wmin = shift < 0 ? int(-shift) : 0;
	uint32_t* const base = jb.out + (shift > 0 ? shift : 0) - wmin;
	int b = 0;
	for (int w0 = 0; w0 < count; w0 += 4 * mm, b ^= 1) {
		if (t < mm) {
			uint32_t w[4];
			half_four(win[b], t, mm, p, w);
			win[b ^ 1][t] = w[2];
			win[b ^ 1][mm + t] = w[3];
			if (w0 >= wmin && w0 + 4 * mm <= count) {
#pragma unroll
				for (int q = 0; q < 4; ++q) base[w0 + q * mm + t] = temper(w[q], p);
			} else {
				for (int q = 0; q < 4; ++q) {
					const int k = w0 + q * mm + t;
					if (k >= wmin && k < count) base[k] = temper(w[q], p);
				}
			}
		}
		__syncthreads();
	}
}

// Window of segment 0 of each jumped job: the seeded state, or a copy of the
// job's own window.
__global__ void mt_seed_kernel(const arma_mt_params* __restrict__ ps,
                               const uint32_t* __restrict__ seeds,
                               const uint32_t* const* __restrict__ src, uint32_t* const* dst) {
	const uint32_t* s = src[blockIdx.x];
	if (s) {
		for (int k = threadIdx.x; k < ps[blockIdx.x].nn; k += blockDim.x) dst[blockIdx.x][k] = s[k];
	} else if (threadIdx.x == 0) {
		seed_state(dst[blockIdx.x], seeds[blockIdx.x], ps[blockIdx.x]);
	}
}

// Inverse of temper(): each xor-shift step y ^= (y >> s) (or (y << s) & mask)
// is undone by the fixed-point iteration x <- y ^ (x >> s), which settles s
// more bits per pass.
__device__ __forceinline__ uint32_t undo_right(uint32_t y, int s) {
	uint32_t x = y;
	for (int k = 0; k < 32; k += s) x = y ^ (x >> s);
	return x;
}
__device__ __forceinline__ uint32_t undo_left(uint32_t y, int s, uint32_t mask) {
	uint32_t x = y;
	for (int k = 0; k < 32; k += s) x = y ^ ((x << s) & mask);
	return x;
}
__device__ __forceinline__ uint32_t untemper(uint32_t y, const arma_mt_params& p) {
	y = undo_right(y, p.shift1);
	y = undo_left(y, p.shiftC, p.maskC);
	y = undo_left(y, p.shiftB, p.maskB);
	return undo_right(y, p.shift0);
}

struct WindowJob {
	arma_mt_params p;
	const uint32_t* words;               // tempered words of the last chunk
	unsigned long long n_words;          // words generated for it
	const unsigned long long* attempts;  // polar attempts the chunk consumed
	uint32_t* window;                    // raw window at the next word
	unsigned long long* position;        // running word position (may be null)
};

// The raw window in front of word 4*attempts: untempered copies of the nn
// words before it.  A chunk whose noise ran short reports no attempt count
// (0): the window is left as it was and the chunk is generated again.
__global__ void mt_window_kernel(const WindowJob* __restrict__ jobs) {
	const WindowJob& jb = jobs[blockIdx.x];
	const unsigned long long used = 4ull * *jb.attempts;
	const int n = jb.p.nn;
	if (used < (unsigned long long)n || used > jb.n_words) return;
	for (int k = threadIdx.x; k < n; k += blockDim.x)
		jb.window[k] = untemper(jb.words[used - n + k], jb.p);
	if (threadIdx.x == 0 && jb.position) *jb.position += used;
}

// The window D ahead of a jump's source: dst[w] = XOR over the set bits i of
// t^D mod phi of y[i + w], y the raw sequence from the source window on.
// `parts` CTAs share a jump (more when few jumps run at once), each a range of
// the bits; its warps share that range again.  A CTA computes the raw words it
// needs into shared memory.  A lane owns kJumpWords consecutive words of the
// window, so that a set bit costs a warp kJumpWords XORs in registers and the
// words that 16 bits touch are read once for all of them (a lane's stride is
// odd: no bank conflicts); two neighbouring set bits go in one three-input XOR.
// At p = 19937: 10 us alone in 32 parts, 1.1 ms for the 2700 jumps of the batch
// of 256 surfaces (one word per thread and a shared-memory read per set bit: 45
// us alone, 4.3 ms).
constexpr int kJumpWords = 21;                // 32 * 21 = 672 >= 624 words
constexpr int kJumpSpan = 32 * kJumpWords;    // words of the window per pass
constexpr int kJumpBits = 16;                 // bits whose words are read together

__host__ __device__ inline int jump_degree(const arma_mt_params& p) { return 32 * p.nn - p.rr; }
// raw words a jump can read: bits up to the degree, rounded up to whole groups,
// plus the window's passes
__host__ __device__ inline int jump_words(const arma_mt_params& p) {
	const int passes = (p.nn + kJumpSpan - 1) / kJumpSpan;
	return (jump_degree(p) + kJumpBits) / kJumpBits * kJumpBits + passes * kJumpSpan + kJumpBits;
}

__global__ void __launch_bounds__(kJumpThreads)
mt_jump_kernel(const JumpJob* __restrict__ jobs, int parts) {
	extern __shared__ uint32_t y[];
	const JumpJob& jb = jobs[blockIdx.x / parts];
	const arma_mt_params p = in_registers(jb.p);
	const int n = p.nn, m = p.mm, chunk = n - m;
	const int groups = (jump_degree(p) + kJumpBits - 1) / kJumpBits;
	const int per = (groups + parts - 1) / parts;
	const int g0 = min(groups, int(blockIdx.x % parts) * per), g1 = min(groups, g0 + per);
	if (g0 >= g1) return;  // uniform over the CTA
	const int len = min(jump_words(p), g1 * kJumpBits + (n + kJumpSpan - 1) / kJumpSpan * kJumpSpan);
	for (int k = threadIdx.x; k < n; k += blockDim.x) y[k] = jb.src[k];
	__syncthreads();
	if (half_set(p)) {
		for (int j0 = 0; j0 + n < len; j0 += 4 * m) {
			const int t = threadIdx.x;
			if (t < m) {
				uint32_t w[4];
				half_four(y + j0, t, m, p, w);
#pragma unroll
				for (int q = 0; q < 4; ++q)
					if (j0 + n + q * m + t < len) y[j0 + n + q * m + t] = w[q];
			}
			__syncthreads();
		}
	} else {
		for (int j0 = n; j0 < len; j0 += chunk) {
			for (int t = threadIdx.x; t < chunk; t += blockDim.x)
				if (j0 + t < len) y[j0 + t] = y[j0 + t - chunk] ^ twist(y[j0 + t - n], y[j0 + t - n + 1], p);
			__syncthreads();
		}
	}
	__shared__ uint32_t sum[kJumpSpan];
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	constexpr int kWarps = kJumpThreads / 32;
	const auto* pattern = reinterpret_cast<const uint16_t*>(jb.bits);  // little endian
	for (int w0 = 0; w0 < n; w0 += kJumpSpan) {
		for (int k = threadIdx.x; k < kJumpSpan; k += blockDim.x) sum[k] = 0u;
		__syncthreads();
		uint32_t acc[kJumpWords];
#pragma unroll
		for (int r = 0; r < kJumpWords; ++r) acc[r] = 0u;
		for (int g = g0 + warp; g < g1; g += kWarps) {
			const uint32_t pat = __shfl_sync(0xffffffffu, uint32_t(pattern[g]), 0);
			const uint32_t* src = y + g * kJumpBits + w0 + lane * kJumpWords;
			uint32_t v[kJumpWords + kJumpBits - 1];
#pragma unroll
			for (int r = 0; r < kJumpWords + kJumpBits - 1; ++r) v[r] = src[r];
#pragma unroll
			for (int k = 0; k < kJumpBits; k += 2) {
				const uint32_t two = (pat >> k) & 3u;
				if (two == 3u) {
#pragma unroll
					for (int r = 0; r < kJumpWords; ++r) acc[r] ^= v[k + r] ^ v[k + 1 + r];
				} else if (two == 1u) {
#pragma unroll
					for (int r = 0; r < kJumpWords; ++r) acc[r] ^= v[k + r];
				} else if (two == 2u) {
#pragma unroll
					for (int r = 0; r < kJumpWords; ++r) acc[r] ^= v[k + 1 + r];
				}
			}
		}
#pragma unroll
		for (int r = 0; r < kJumpWords; ++r) atomicXor(&sum[lane * kJumpWords + r], acc[r]);
		__syncthreads();
		for (int k = threadIdx.x; k < kJumpSpan && w0 + k < n; k += blockDim.x) {
			if (parts > 1) atomicXor(&jb.dst[w0 + k], sum[k]);
			else jb.dst[w0 + k] = sum[k];
		}
		__syncthreads();
	}
}

std::vector<uint32_t> params_key(const arma_mt_params& p) {
	std::vector<uint32_t> k(sizeof(p) / 4);
	std::memcpy(k.data(), &p, sizeof(p));
	k.back() = 0;  // the `i` field does not affect the stream
	return k;
}

// Jump tables on the device are cached per (device, parameter set, exponent)
// for the life of the process; every context on the device shares them.
std::mutex g_table_mutex;
std::map<std::vector<uint32_t>, uint32_t*> g_tables;

// The device's t^(2^e) mod phi of a set, or null when there is no such phi.
const uint32_t* jump_table(Ctx* c, const arma_mt_params& p, int e) {
	auto key = params_key(p);
	key.push_back(uint32_t(c->device));
	key.push_back(uint32_t(e));
	std::lock_guard<std::mutex> lock(g_table_mutex);
	auto it = g_tables.find(key);
	if (it != g_tables.end()) return it->second;
	std::vector<uint32_t> bits;
	uint32_t* d = nullptr;
	if (mt_jump_bits(p, e, &bits)) {
		ARMA_CUDA_TRY(cudaMalloc(&d, sizeof(uint32_t) * bits.size()));
		ARMA_CUDA_TRY(cudaMemcpy(d, bits.data(), sizeof(uint32_t) * bits.size(),
		                         cudaMemcpyHostToDevice));
	}
	return g_tables.emplace(key, d).first->second;
}

// Dynamic shared memory a jump can have: the CTA's most less the kernel's sums.
constexpr size_t kJumpSmem = kSmemOptin - sizeof(uint32_t) * kJumpSpan;
size_t jump_smem(const arma_mt_params& p) { return sizeof(uint32_t) * size_t(jump_words(p)); }

// Streams up to this length stay one segment: 85 us for its one CTA.
constexpr unsigned long long kWhole = 1ull << 18;

// Segments of a stream cut at 2^v words, v <= log2_seg.
unsigned long long segments_of(unsigned long long total, int v, int log2_seg) {
	if (total <= std::min(kWhole, 1ull << log2_seg)) return 1;
	return (total + (1ull << v) - 1) >> v;
}

// The segment length of a call, 2^v words with v at most the caller's: the
// shortest that still gives no more than four segments per SM.  Generating a
// segment takes one CTA 0.41 us per 1248 words and another level of the jump
// tree 10 us, so a single stream is cut short (16.7 M words in 256 segments: 260
// us; 16 segments of 2^20, a warp each: 1130 us), while the jumps of a large
// batch keep its segments long (2.7 G words, 2700 segments of 2^20).
int segment_log2(Ctx* c, const std::vector<MtJob>& jobs, int log2_seg) {
	auto count = [&](int v) {
		unsigned long long n = 0;
		for (const MtJob& j : jobs) n += segments_of(j.offset + j.count, v, log2_seg);
		return n;
	};
	int v = log2_seg;
	while (v > kMinLog2Seg && count(v - 1) <= 4ull * c->num_sms) --v;
	return v;
}

}  // namespace

namespace {
// The jump-ahead windows and the generation of a batch of jobs.  prepare:
// only the windows (at every segment start of every job longer than one
// segment), handed back in prepare[q].seg_states; a job that already carries
// seg_states is not jumped again.
void mt_batch(Ctx* c, const std::vector<MtJob>& jobs, int log2_seg, std::vector<MtJob>* prepare) {
	ProfScope prof_(c, "mt");
	ARMA_REQUIRE(log2_seg >= 12 && log2_seg <= 24, ARMA_EINVAL, "bad MT segment length");
	for (const MtJob& j : jobs) {
		ARMA_REQUIRE(!j.state || j.offset == 0, ARMA_EINVAL,
		             "an MT job started from a window has no offset");
		ARMA_REQUIRE(j.p.nn > 1 && j.p.mm > 0 && j.p.mm < j.p.nn && j.p.ww == 32, ARMA_EINVAL,
		             "bad MT parameter set");
		ARMA_REQUIRE(j.p.nn + (j.p.nn - j.p.mm) <= kRing &&
		                 j.p.nn - j.p.mm <= kMaxOwn * kGenMaxThreads,
		             ARMA_EINVAL, "MT state too large for the device generator");
	}
	if (jobs.empty()) return;
	const int v_call = segment_log2(c, jobs, log2_seg);
	// segments per job, 2^v[q] words each; jobs with more than one need jumps
	std::vector<int> K(jobs.size()), v(jobs.size(), v_call);
	int Kmax = 1;
	size_t nstates = 0;
	std::vector<char> ready(jobs.size(), 0);  // windows precomputed: no jumps here
	std::vector<const uint32_t*> state0(jobs.size(), nullptr);  // per job: K windows of nn words
	for (size_t q = 0; q < jobs.size(); ++q) {
		const unsigned long long total = jobs[q].offset + jobs[q].count;
		ARMA_REQUIRE(segments_of(total, log2_seg, log2_seg) <= (1ull << kLevels), ARMA_EINVAL,
		             "MT stream too long");
		if (jobs[q].seg_states) {
			v[q] = jobs[q].seg_log2;
			K[q] = int(segments_of(total, v[q], log2_seg));
			ARMA_REQUIRE(K[q] > 1, ARMA_EINVAL, "MT job with windows but one segment");
			ready[q] = 1;
			state0[q] = jobs[q].seg_states;
			continue;
		}
		K[q] = int(segments_of(total, v[q], log2_seg));
		// one sequential segment where the jump's words do not fit in shared memory
		// or no polynomial of the state's degree was found
		if (K[q] > 1 && (jump_smem(jobs[q].p) > kJumpSmem || !jump_table(c, jobs[q].p, v[q]))) K[q] = 1;
		if (K[q] > 1) nstates += size_t(K[q]) * jobs[q].p.nn;
		if (K[q] > 1) Kmax = std::max(Kmax, K[q]);
	}
	if (nstates) {
		uint32_t* states = static_cast<uint32_t*>(scratch_take(c, sizeof(uint32_t) * nstates));
		ARMA_CUDA_TRY(cudaMemsetAsync(states, 0, sizeof(uint32_t) * nstates, c->stream));
		size_t off = 0;
		std::vector<arma_mt_params> ps;
		std::vector<uint32_t> seeds;
		std::vector<const uint32_t*> src;
		std::vector<uint32_t*> dst;
		for (size_t q = 0; q < jobs.size(); ++q) {
			if (K[q] <= 1 || ready[q]) continue;
			state0[q] = states + off;
			off += size_t(K[q]) * jobs[q].p.nn;
			ps.push_back(jobs[q].p);
			seeds.push_back(jobs[q].seed);
			src.push_back(jobs[q].state);
			dst.push_back(states + (state0[q] - states));
		}
		auto* d_ps = static_cast<arma_mt_params*>(scratch_take(c, sizeof(arma_mt_params) * ps.size()));
		auto* d_seeds = static_cast<uint32_t*>(scratch_take(c, sizeof(uint32_t) * seeds.size()));
		auto* d_src = static_cast<const uint32_t**>(scratch_take(c, sizeof(uint32_t*) * src.size()));
		auto* d_dst = static_cast<uint32_t**>(scratch_take(c, sizeof(uint32_t*) * dst.size()));
		ARMA_CUDA_TRY(copy_async(c, d_ps, ps.data(), sizeof(arma_mt_params) * ps.size(),
		                              cudaMemcpyHostToDevice, c->stream));
		ARMA_CUDA_TRY(copy_async(c, d_seeds, seeds.data(), sizeof(uint32_t) * seeds.size(),
		                              cudaMemcpyHostToDevice, c->stream));
		ARMA_CUDA_TRY(copy_async(c, d_src, src.data(), sizeof(uint32_t*) * src.size(),
		                              cudaMemcpyHostToDevice, c->stream));
		ARMA_CUDA_TRY(copy_async(c, d_dst, dst.data(), sizeof(uint32_t*) * dst.size(),
		                              cudaMemcpyHostToDevice, c->stream));
		// binary tree of jumps, widest stride first; every level's jumps in one
		// table
		int levels = 0;
		while ((1 << levels) < Kmax) ++levels;
		size_t smem = 0;
		for (size_t q = 0; q < jobs.size(); ++q)
			if (K[q] > 1 && !ready[q])
				smem = std::max(smem, jump_smem(jobs[q].p));
		std::vector<JumpJob> jj;
		std::vector<size_t> level_at(levels + 1, 0);  // level lv: entries from level_at[lv + 1] on
		for (int lv = levels - 1; lv >= 0; --lv) {
			level_at[lv + 1] = jj.size();
			const int step = 1 << lv;
			for (size_t q = 0; q < jobs.size(); ++q) {
				if (K[q] <= 1 || ready[q]) continue;
				const int nn = jobs[q].p.nn;
				uint32_t* w = states + (state0[q] - states);
				const uint32_t* bits = step < K[q] ? jump_table(c, jobs[q].p, v[q] + lv) : nullptr;
				for (int base = 0; base + step < K[q]; base += 2 * step)
					jj.push_back(JumpJob{jobs[q].p, w + size_t(base) * nn,
					                     w + size_t(base + step) * nn, bits});
			}
		}
		level_at[0] = jj.size();
		auto* d_jj = static_cast<JumpJob*>(scratch_take(c, sizeof(JumpJob) * jj.size()));
		ARMA_CUDA_TRY(copy_async(c, d_jj, jj.data(), sizeof(JumpJob) * jj.size(),
		                              cudaMemcpyHostToDevice, c->stream));
		mt_seed_kernel<<<int(ps.size()), 32, 0, c->stream>>>(d_ps, d_seeds, d_src, d_dst);
		c->launches += 1;
		allow_smem(mt_jump_kernel, smem, sizeof(uint32_t) * kJumpSpan);
		for (int lv = levels - 1; lv >= 0; --lv) {
			const size_t at = level_at[lv + 1], n = level_at[lv] - at;
			if (n == 0) continue;
			// few jumps at this level: split each over several CTAs, at most 32
			// (a CTA first runs the recurrence up to its bits, about 4 us)
			const int parts = int(std::min<size_t>(32, std::max<size_t>(1, 2 * size_t(c->num_sms) / n)));
			mt_jump_kernel<<<unsigned(n) * parts, kJumpThreads, smem, c->stream>>>(d_jj + at, parts);
			ARMA_CUDA_TRY(cudaGetLastError());
			c->launches += 1;
		}
	}
	if (prepare) {
		for (size_t q = 0; q < jobs.size(); ++q)
			if (K[q] > 1) {
				(*prepare)[q].seg_states = state0[q];
				(*prepare)[q].seg_log2 = v[q];
			}
		return;
	}
	// generation: one CTA or warp per segment
	std::vector<SegJob> seg;
	for (size_t q = 0; q < jobs.size(); ++q) {
		const unsigned long long total = jobs[q].offset + jobs[q].count, J = 1ull << v[q];
		for (int k = 0; k < K[q]; ++k) {
			const unsigned long long first = (unsigned long long)k * J;
			if (K[q] > 1 && first + J <= jobs[q].offset) continue;  // entirely skipped
			SegJob s;
			s.p = jobs[q].p;
			s.seed = jobs[q].seed;
			s.state = K[q] > 1 ? state0[q] + size_t(k) * jobs[q].p.nn : jobs[q].state;
			s.first = first;
			s.count = K[q] > 1 ? std::min(J, total - first) : total;
			s.offset = jobs[q].offset;
			s.out = jobs[q].out;
			seg.push_back(s);
		}
	}
	// segments of nn = 2 mm sets (32-bit word indices): one warp each when there
	// are many, one CTA each when they are few; the others one CTA each in the
	// general form
	auto half = [&](const SegJob& j) {
		return half_set(j.p) && j.count < (1ull << 30) &&
		       j.offset < (1ull << 30) && j.first < (1ull << 40);
	};
	std::stable_partition(seg.begin(), seg.end(), half);
	const int nhalf = int(std::count_if(seg.begin(), seg.end(), half));
	const bool by_warp = size_t(nhalf) > kWarpSegments * size_t(c->num_sms);
	auto* d_seg = static_cast<SegJob*>(scratch_take(c, sizeof(SegJob) * seg.size()));
	ARMA_CUDA_TRY(copy_async(c, d_seg, seg.data(), sizeof(SegJob) * seg.size(),
	                              cudaMemcpyHostToDevice, c->stream));
	if (nhalf > 0 && !by_warp) {
		mt_generate_four_kernel<<<nhalf, kFourThreads, 0, c->stream>>>(d_seg);
		ARMA_CUDA_TRY(cudaGetLastError());
		c->launches += 1;
	} else if (nhalf > 0) {
		// mm = 312 (the sets of period 2^19937 - 1) compiled in; others at run time
		bool all312 = true;
		for (int k = 0; k < nhalf; ++k) all312 = all312 && seg[k].p.mm == 312;
		const int hgrid = (nhalf + kHalfWarps - 1) / kHalfWarps;
		if (all312)
			mt_generate_half_kernel<312><<<hgrid, 32 * kHalfWarps, 0, c->stream>>>(d_seg, nhalf);
		else
			mt_generate_half_kernel<0><<<hgrid, 32 * kHalfWarps, 0, c->stream>>>(d_seg, nhalf);
		ARMA_CUDA_TRY(cudaGetLastError());
		c->launches += 1;
	}
	const int grid = int(seg.size()) - nhalf;
	if (grid > 0) {
		int chunk = 1;  // the largest chunk of the rest
		for (size_t k = size_t(nhalf); k < seg.size(); ++k)
			chunk = std::max(chunk, seg[k].p.nn - seg[k].p.mm);
		const int threads = std::min(kGenMaxThreads, (chunk + 31) / 32 * 32);
		const int own = (chunk + threads - 1) / threads;
		const SegJob* rest = d_seg + nhalf;
		switch (own) {
			case 1: mt_generate_kernel<1><<<grid, threads, 0, c->stream>>>(rest); break;
			case 2: mt_generate_kernel<2><<<grid, threads, 0, c->stream>>>(rest); break;
			case 3: mt_generate_kernel<3><<<grid, threads, 0, c->stream>>>(rest); break;
			default: mt_generate_kernel<4><<<grid, threads, 0, c->stream>>>(rest); break;
		}
		ARMA_CUDA_TRY(cudaGetLastError());
		c->launches += 1;
	}
}

}  // namespace

void launch_mt_generate_batch(Ctx* c, const std::vector<MtJob>& jobs, int log2_seg) {
	mt_batch(c, jobs, log2_seg, nullptr);
}

void launch_mt_prepare(Ctx* c, std::vector<MtJob>& jobs, int log2_seg) {
	mt_batch(c, jobs, log2_seg, &jobs);
}

void launch_mt_window_update(Ctx* c, const std::vector<MtWindowSpec>& specs) {
	if (specs.empty()) return;
	ProfScope prof_(c, "mt");
	std::vector<WindowJob> jobs(specs.size());
	for (size_t k = 0; k < specs.size(); ++k)
		jobs[k] = WindowJob{specs[k].p, specs[k].words, specs[k].n_words, specs[k].attempts,
		                    specs[k].window, specs[k].position};
	auto* d_jobs = static_cast<WindowJob*>(scratch_take(c, sizeof(WindowJob) * jobs.size()));
	ARMA_CUDA_TRY(copy_async(c, d_jobs, jobs.data(), sizeof(WindowJob) * jobs.size(),
	                              cudaMemcpyHostToDevice, c->stream));
	mt_window_kernel<<<int(jobs.size()), 256, 0, c->stream>>>(d_jobs);
	ARMA_CUDA_TRY(cudaGetLastError());
	c->launches += 1;
}

void launch_mt_generate(Ctx* c, const arma_mt_params& p, uint32_t seed,
                        uint64_t offset, uint64_t n, uint32_t* d_out) {
	if (n == 0) return;
	launch_mt_generate_batch(c, {MtJob{p, seed, offset, n, d_out}});
	// the job tables live in scratch and pageable host vectors: finish first
	ARMA_CUDA_TRY(cudaStreamSynchronize(c->stream));
}

}  // namespace armab
