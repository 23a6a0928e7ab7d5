// Host-side GF(2) polynomial arithmetic for jumping a dcmt Mersenne Twister
// stream ahead.
//
// The essential state of a w=32 dcmt generator has p = 32*nn - rr bits and
// evolves by an invertible linear map A over GF(2).  Every bit of the raw
// word sequence x[j] (sgenrand_mt's state followed by the recurrence) is a
// fixed linear functional of the state, so all of them satisfy the
// characteristic polynomial phi(t) of A.  For a jump of J words:
//     g(t) = t^J mod phi(t)   =>   x[J + w] = XOR_{i : g_i = 1} x[i + w]
// for w >= 1 (and the upper 32-rr bits of w = 0), i.e. the window of nn words
// J positions ahead is an XOR of windows of the raw sequence.  phi is the closed
// form of dcmt.cpp, checked against the sequence (Berlekamp-Massey on 2p bits of
// one bit position where the masks are not a dcmt set's); t^J for J = 2^q comes
// from q modular squarings.  A set's first tables take about 6 ms at p = 19937
// (170 ms with Berlekamp-Massey and bitwise reductions).
#include <algorithm>
#include <cstdint>
#include <cstring>
#include <map>
#include <mutex>
#include <vector>

#include "internal.h"

namespace armab {
namespace {

using Bits = std::vector<uint64_t>;

inline int get_bit(const Bits& b, long i) { return int((b[size_t(i) >> 6] >> (i & 63)) & 1u); }
inline void flip_bit(Bits& b, long i) { b[size_t(i) >> 6] ^= uint64_t(1) << (i & 63); }

// 64 bits of b starting at bit `off` (bits beyond the end read as 0).
inline uint64_t word_at(const Bits& b, long off) {
	const size_t w = size_t(off) >> 6;
	const int s = int(off & 63);
	const uint64_t lo = w < b.size() ? b[w] : 0;
	if (s == 0) return lo;
	const uint64_t hi = (w + 1) < b.size() ? b[w + 1] : 0;
	return (lo >> s) | (hi << (64 - s));
}

// a ^= b << sh  (a sized to hold the result)
void xor_shifted(Bits& a, const Bits& b, long sh, long nbits_b) {
	const size_t ws = size_t(sh) >> 6;
	const int bs = int(sh & 63);
	const size_t nw = (size_t(nbits_b) + 63) >> 6;
	for (size_t i = 0; i < nw; ++i) {
		const uint64_t v = i < b.size() ? b[i] : 0;
		if (ws + i < a.size()) a[ws + i] ^= v << bs;
		if (bs && ws + i + 1 < a.size()) a[ws + i + 1] ^= v >> (64 - bs);
	}
}

// Raw words x[0..count) of the dcmt recurrence from the seeded state.
std::vector<uint32_t> raw_words(const arma_mt_params& p, uint32_t seed, size_t count) {
	const int n = p.nn, m = p.mm;
	std::vector<uint32_t> x(count);
	uint32_t s = seed;
	for (int k = 0; k < n && size_t(k) < count; ++k) {
		x[k] = s & p.wmask;
		s = 1812433253u * (s ^ (s >> 30)) + uint32_t(k + 1);
	}
	for (size_t j = n; j < count; ++j) {
		const uint32_t y = (x[j - n] & p.umask) | (x[j - n + 1] & p.lmask);
		x[j] = x[j - n + m] ^ (y >> 1) ^ ((y & 1u) ? p.aaa : 0u);
	}
	return x;
}

// Berlekamp-Massey over GF(2).  Returns the characteristic polynomial (bit i
// = coefficient of t^i) and its degree.
Bits berlekamp_massey(const std::vector<uint8_t>& s, int* degree) {
	const long N = long(s.size());
	const size_t nw = size_t(N + 64) / 64 + 1;
	Bits C(nw, 0), B(nw, 0), T;
	C[0] = B[0] = 1;
	// reversed sequence: r bit j = s[N-1-j], so s[n-i] = r[(N-1-n) + i]
	Bits r(nw, 0);
	for (long j = 0; j < N; ++j)
		if (s[N - 1 - j]) flip_bit(r, j);
	long L = 0, m = 1;
	for (long n = 0; n < N; ++n) {
		// d = s[n] + sum_{i=1..L} C_i s[n-i] = parity(C & r>>(N-1-n)) over bits 0..L
		uint64_t acc = 0;
		const long base = N - 1 - n;
		const size_t words = size_t(L + 64) / 64;
		for (size_t w = 0; w < words; ++w) {
			uint64_t c = C[w];
			if (w == words - 1) {
				const int rem = int((L + 1) - long(w) * 64);
				if (rem < 64) c &= (uint64_t(1) << rem) - 1;
			}
			acc ^= c & word_at(r, base + long(w) * 64);
		}
		const int d = __builtin_parityll(acc);
		if (d == 0) {
			++m;
		} else if (2 * L <= n) {
			T = C;
			xor_shifted(C, B, m, long(B.size()) * 64);
			L = n + 1 - L;
			B = T;
			m = 1;
		} else {
			xor_shifted(C, B, m, long(B.size()) * 64);
			++m;
		}
	}
	// phi(t) = t^L C(1/t): coefficient of t^(L-i) is C_i
	Bits phi(size_t(L) / 64 + 1, 0);
	for (long i = 0; i <= L; ++i)
		if (get_bit(C, i)) flip_bit(phi, L - i);
	*degree = int(L);
	return phi;
}

// A parameter set's powers t^(2^e) mod phi, e = 0, 1, ...: found once, extended
// as larger exponents are asked for.
struct JumpPowers {
	Bits phi;             // empty: no polynomial of the state's degree
	std::vector<Bits> g;  // g[e] = t^(2^e) mod phi
};

// Whether phi annihilates the sequence: 64 windows of words from a seeded state,
// 2048 bit positions.
bool annihilates(const Bits& phi, int p, const std::vector<uint32_t>& x, size_t start) {
	for (size_t w = 0; w < 64; ++w) {
		uint32_t v = 0;
		for (int i = 0; i <= p; ++i)
			if (get_bit(phi, i)) v ^= x[start + w + size_t(i)];
		if (v) return false;
	}
	return true;
}

JumpPowers find_powers(const arma_mt_params& prm) {
	JumpPowers r;
	const int p = 32 * prm.nn - prm.rr;
	// past the seeded words, whose first has bits outside the state
	const size_t start = size_t(prm.nn);
	const std::vector<uint32_t> x = raw_words(prm, 4357u, start + 2 * size_t(p) + 64);
	r.phi = dcmt::characteristic_polynomial(prm);
	if (r.phi.empty() || !annihilates(r.phi, p, x, start)) {
		// masks of another shape: the minimal polynomial of 2p bits of one bit
		// position
		std::vector<uint8_t> s(2 * size_t(p));
		for (size_t j = 0; j < s.size(); ++j) s[j] = uint8_t(x[start + j] & 1u);
		int L = 0;
		r.phi = berlekamp_massey(s, &L);
		if (L != p) {  // the caller generates sequentially
			r.phi.clear();
			return r;
		}
	}
	Bits t(size_t(p) / 64 + 1, 0);
	flip_bit(t, 1);
	r.g.push_back(std::move(t));
	return r;
}

std::mutex g_powers_mutex;
std::map<std::vector<uint32_t>, JumpPowers> g_powers;

}  // namespace

bool mt_jump_bits(const arma_mt_params& prm, int e, std::vector<uint32_t>* bits) {
	std::vector<uint32_t> key(sizeof(prm) / 4);
	std::memcpy(key.data(), &prm, sizeof(prm));
	key.back() = 0;  // the `i` field does not affect the stream
	std::lock_guard<std::mutex> lock(g_powers_mutex);
	auto it = g_powers.find(key);
	if (it == g_powers.end()) it = g_powers.emplace(key, find_powers(prm)).first;
	JumpPowers& jp = it->second;
	if (jp.phi.empty()) return false;
	const int p = 32 * prm.nn - prm.rr;
	if (int(jp.g.size()) <= e) dcmt::square_powers_of_t(jp.phi, p, int(jp.g.size()), e, &jp.g);
	bits->assign((size_t(p) + 31) / 32, 0u);
	for (long i = 0; i < p; ++i)
		if (get_bit(jp.g[e], i)) (*bits)[size_t(i) >> 5] |= 1u << (i & 31);
	return true;
}

}  // namespace armab
