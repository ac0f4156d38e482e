// Attention of a prompt behind cached tokens with an additive mask [b, 1, t, S], head size 128, fp16: what QuantLlamaAttention.forward does between
// its two projections.
//
//   attn_prepare_kernel  classifies the 64 x 64 tiles of the mask (nothing visible / low / mixed / zero), writes the low and mixed ones in the order in which the
//                        other kernel's threads hold them, and copies the cached rows in front of the new ones, which the projection writes in place:
//                        no concatenation
//   attn_prompt_kernel   one CTA of four warps per head and 64 queries; keys and values in tiles of 64, fetched asynchronously two deep; products on
//                        mma.m16n8k16, scores, softmax and sums in fp32.  Tiles in which nothing is visible are neither loaded nor computed, and
//                        the mask is read for mixed tiles only, so a causal mask costs half of the products and its diagonal.
//
// Causal masks come with minus infinity or with a large negative number (the lowest fp16 value).  A tile whose entries are all at or below AP_LOW_MAX is left
// for last, and left out when no key in it can matter: with |score| <= |q| |k| scale, every weight of the tile is below 2^-200 of what the
// row has seen, which is zero in fp32 and changes no bit of the result (finite values assumed).  The largest |k|^2 of a tile is computed by the first
// CTA that asks and kept in the scratch for the others.  Rows that see nothing but such tiles compute them.  The lowest value / minus infinity, this kernel, 32 heads,
// us: 701 behind 64 25 / 25, 2047 125 / 121, 3001 258 / 254; with all masked tiles computed (two-byte loads of the mask) 53 / 25, 296 / 124, 626 / 252.  Low and mixed
// tiles come by the asynchronous copies of their keys: biases everywhere, whole layer, 2047 506 -> 489, library 480.
//
// What bounds it: issue and latency of the legacy tensor path with eight warps per SM, so a library kernel on the tcgen05 path is
// the better one for long prompts whose mask rows start on 16 bytes; the rule stands in csrc/host/calls.cpp.  Two blocks of 16 queries per warp, which read keys and values
// half as often, were slower (255 registers: 701 queries behind 64, 32 heads 51.6 us; one block 35.7; mask copy, concatenation and library kernel 59).
// Under a causal mask the last queries have the longest rows of tiles, so the CTAs of all heads start with those: head by head, the last heads' long CTAs started when
// the chip was emptying (tensor pipe 25 % busy on average, 37 % on the busiest SM).  Whole layer, us: 701 behind 64 119.4 -> 112.6, 1300 behind 3 250 -> 241.
// Long ones first and then from the shortest up: 116.
#include <algorithm>

#include "common.cuh"

namespace gptq {

bool pdl_enabled();          // api.cu

namespace {

constexpr int AP_D = 128, AP_T = 64, AP_THREADS = 128;
constexpr int AP_TILE = AP_T * AP_D * 2;                 // bytes of a tile of queries, keys or values
constexpr int AP_MASK = AP_T * AP_T * 2;                 // ... of the mask
constexpr float AP_LOG2E = 1.4426950408889634f;
constexpr float AP_LOW_MAX = -8192.f;
constexpr uint32_t AP_LOW_BITS = 0xF000u;                // the same in fp16; larger bits up to 0xFC00 are lower numbers
enum { AP_HIDDEN = 0, AP_MIXED = 1, AP_OPEN = 2, AP_LOW = 3 };          // AP_LOW with the full scratch only

// The full scratch: classes, largest |k|^2 of every head's key tiles (bits of a float; 0: not known yet), low and mixed tiles of the mask.
struct FullScratch {
	size_t norms, tiles, bytes;
	FullScratch(int mask_b, int b, int heads, int t, int S) {
		const size_t qt = (t + AP_T - 1) / AP_T, kt = (S + AP_T - 1) / AP_T, n = (size_t)mask_b * qt * kt;
		norms = (n + 255) / 256 * 256;
		tiles = norms + ((size_t)b * heads * kt * 4 + 255) / 256 * 256;
		bytes = tiles + n * (AP_T * AP_T * 2);
	}
};

struct PrepareParams {
	const __half *mask;
	long long mask_sb, mask_st;
	int mask_b, t, S, qt, kt;
	unsigned char *flags;                // [mask_b][qt][kt]
	unsigned *norms;                     // full scratch: zeroed here
	uint2 *tiles;                        // full scratch: 64 x 64 entries as [warp][4][lane] x 16 bytes, see attn_prompt_kernel; else NULL
	int n_norms;
	const __half *past_k, *past_v;       // [b, heads, past, 128], rows contiguous
	long long pk_sb, pk_sh, pv_sb, pv_sh;
	int b, heads, past;
	__half *k, *v;                       // [b, heads, S, 128]
	int mask_ctas;
};

__global__ void __launch_bounds__(256) attn_prepare_kernel(const PrepareParams p) {
	pdl_wait();          // both kernels: launch latency only, nothing is read or written ahead
	if ((int)blockIdx.x < p.mask_ctas) {
		// a tile: 256 threads, a quarter of a row each
		const int id = blockIdx.x, kt = id % p.kt, rest = id / p.kt, qt = rest % p.qt, mb = rest / p.qt;
		const int row = qt * AP_T + (threadIdx.x >> 2), col = kt * AP_T + (threadIdx.x & 3) * 16;
		uint32_t e[8], seen = 7u;          // entries in pairs; nothing but -infinity | zeros | -infinity to AP_LOW_MAX
#pragma unroll
		for (int i = 0; i < 8; ++i) e[i] = row < p.t ? 0xFC00FC00u : 0u;          // (columns that do not exist are hidden)
		if (row < p.t) {
			const unsigned short *src = reinterpret_cast<const unsigned short *>(p.mask) + mb * p.mask_sb + row * p.mask_st + col;
#pragma unroll
			for (int i = 0; i < 16; ++i) {
				if (col + i < p.S) {
					const uint32_t m = __ldg(src + i);
					e[i >> 1] = i & 1 ? (e[i >> 1] & 0xFFFFu) | m << 16 : (e[i >> 1] & 0xFFFF0000u) | m;
					seen &= (m == 0xFC00u ? 1u : 0u) | ((m & 0x7FFFu) == 0u ? 2u : 0u) | (m - AP_LOW_BITS <= 0xFC00u - AP_LOW_BITS ? 4u : 0u);          // (NaN is none of them)
				}
			}
		}
		__shared__ uint32_t s_seen[8];
		seen = __reduce_and_sync(0xffffffffu, seen);
		if ((threadIdx.x & 31) == 0) s_seen[threadIdx.x >> 5] = seen;
		__syncthreads();
#pragma unroll
		for (int i = 0; i < 8; ++i) seen &= s_seen[i];
		const bool hidden = seen & 1u, open = seen & 2u, low = (seen & 4u) && p.tiles;
		if (threadIdx.x == 0) p.flags[id] = hidden ? AP_HIDDEN : open ? AP_OPEN : low ? AP_LOW : AP_MIXED;
		if (!p.tiles) return;
		for (long long i = id * 256ll + threadIdx.x; i < p.n_norms; i += p.mask_ctas * 256ll) p.norms[i] = 0u;
		if (hidden || open) return;
		// row r is entry h = r / 8 % 2 of the lanes 4 (r % 8) + 0 .. 3 of warp r / 16; a lane has columns 8 n + 2 tig, + 1 for n = 0 .. 7: four 16-byte units per h pair
		const int r = threadIdx.x >> 2, quarter = threadIdx.x & 3, unit = (r >> 3 & 1) * 2 + (quarter >> 1);
		uint2 *dst = p.tiles + ((size_t)id * 16 + (r >> 4) * 4 + unit) * 64 + (quarter & 1);
#pragma unroll
		for (int tig = 0; tig < 4; ++tig)
			dst[((r & 7) * 4 + tig) * 2] = make_uint2(e[tig], e[4 + tig]);
		return;
	}
	// cached rows: 16 bytes per thread, keys then values
	const long long half = (long long)p.b * p.heads * p.past * 16;
	for (long long u = (long long)(blockIdx.x - p.mask_ctas) * 256 + threadIdx.x; u < 2 * half; u += (long long)(gridDim.x - p.mask_ctas) * 256) {
		const bool value = u >= half;
		const long long w = value ? u - half : u, c = w & 15, r = (w >> 4) % p.past, h = (w >> 4) / p.past % p.heads, bi = (w >> 4) / p.past / p.heads;
		const __half *src = value ? p.past_v + bi * p.pv_sb + h * p.pv_sh : p.past_k + bi * p.pk_sb + h * p.pk_sh;
		reinterpret_cast<uint4 *>((value ? p.v : p.k) + ((bi * p.heads + h) * p.S + r) * AP_D)[c] = __ldg(reinterpret_cast<const uint4 *>(src + r * AP_D) + c);
	}
}

struct PromptParams {
	const __half *q, *k, *v, *mask;
	long long q_sb, q_st, q_sh, mask_sb, mask_st;
	const unsigned char *flags;
	unsigned *norms;
	const uint4 *tiles;
	__half *out;                         // [b, t, heads * 128]
	int mask_b, heads, t, S, qt, kt;
	float scale;
};

__device__ __forceinline__ void ap_copy16(uint32_t dst, const void *src, bool live) {
	asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void ap_ldmatrix4(uint32_t (&r)[4], uint32_t addr) {
	asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ap_ldmatrix4_trans(uint32_t (&r)[4], uint32_t addr) {
	asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ float ap_exp2(float v) {
	float r;
	asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
	return r;
}
// byte of 16-byte unit u in row r of a tile (256-byte rows; eight neighbouring rows use different banks)
__device__ __forceinline__ uint32_t ap_at(int r, int u) { return (uint32_t)(r * 256 + ((u ^ (r & 7)) << 4)); }

// Largest |k|^2 of up to 64 keys, as the bits of a float (NaN stays above everything); a warp, two keys per lane.
__device__ __noinline__ unsigned ap_key_norm(const __half *k, int rows) {
	unsigned best = 1u;                      // (0 means not known)
	for (int r = threadIdx.x & 31; r < rows; r += 32) {
		float s = 0.f;
#pragma unroll 8
		for (int u = 0; u < AP_D / 8; ++u) {
			const uint4 v = __ldcg(reinterpret_cast<const uint4 *>(k + (size_t)r * AP_D) + u);
			const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
			for (int i = 0; i < 4; ++i) {
				const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&w[i]));
				s = fmaf(f.x, f.x, fmaf(f.y, f.y, s));
			}
		}
		best = max(best, __float_as_uint(s));
	}
	return __reduce_max_sync(0xffffffffu, best);
}

// FULL: with the full scratch.  Without it, `flags` may be NULL (nothing classified) and mixed tiles read the mask itself.
template <bool FULL>
__global__ void __launch_bounds__(AP_THREADS, 2) attn_prompt_kernel(const PromptParams p) {
	extern __shared__ __align__(128) unsigned char ap_smem[];      // K, V of two tiles; queries; FULL: the mask of two tiles
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, gid = lane >> 2, tig = lane & 3;
	const int pairs = gridDim.x / p.qt, late = blockIdx.x / pairs, pair = blockIdx.x - late * pairs;          // the longest of all heads first
	const int qt = p.qt - 1 - late, bi = pair / p.heads, head = pair - bi * p.heads;
	const int q0 = qt * AP_T, mb = p.mask_b == 1 ? 0 : bi;
	const uint32_t base = smem_u32(ap_smem), sq = base + 4 * AP_TILE, sm = sq + AP_TILE + warp * 2048 + lane * 16;
	pdl_wait();
	const __half *q = p.q + bi * p.q_sb + head * p.q_sh, *k = p.k + (size_t)(bi * p.heads + head) * p.S * AP_D, *v = p.v + (size_t)(bi * p.heads + head) * p.S * AP_D;
	const unsigned char *flags = p.flags ? p.flags + ((size_t)mb * p.qt + qt) * p.kt : nullptr;
	const __half *mask = p.mask + mb * p.mask_sb;

	// a tile of 64 rows x 16 units: 8 units per thread
	auto load = [&](uint32_t dst, const __half *src, long long stride, int row0, int rows) {
#pragma unroll
		for (int i = 0; i < 8; ++i) {
			const int e = tid + i * AP_THREADS, r = e >> 4, u = e & 15;
			ap_copy16(dst + ap_at(r, u), src + (row0 + r < rows ? row0 + r : 0) * stride + u * 8, row0 + r < rows);
		}
	};
	bool any_low = false, last = false;          // low tiles have been passed over; they are being computed
	int found = AP_MIXED;                        // class of the tile that next() gave
	auto next = [&](int t) {
		for (; t < p.kt && flags; ++t) {
			found = flags[t];
			if (FULL && found == AP_LOW) any_low = true;
			if (FULL ? found != AP_HIDDEN && (found == AP_LOW) == last : found != AP_HIDDEN) break;
		}
		return t;
	};
	load(sq, q, p.q_st, q0, p.t);
	int cur = next(0), buf = 0;
	// keys, values and, where there is something to add, this thread's share of the mask: tile t, of class `found`, into buffer b
	auto fetch = [&](int t, int b) {
		if (t < p.kt) {
			const uint32_t dst = base + b * 2 * AP_TILE;
			load(dst, k, AP_D, t * AP_T, p.S);
			load(dst + AP_TILE, v, AP_D, t * AP_T, p.S);
			if (FULL && found != AP_OPEN) {
				const uint4 *src = p.tiles + (((size_t)mb * p.qt + qt) * p.kt + t) * (AP_MASK / 16) + warp * 128 + lane;
#pragma unroll
				for (int i = 0; i < 4; ++i) ap_copy16(sm + b * AP_MASK + i * 512, src + i * 32, true);
			}
		}
		cp_async_commit();
	};
	fetch(cur, buf);

	float o[16][4];
#pragma unroll
	for (int n = 0; n < 16; ++n) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f;
	float mx[2] = {-INFINITY, -INFINITY}, sum[2] = {0.f, 0.f};
	const int row = q0 + warp * 16 + gid;      // of o[.][0 .. 1]; row + 8 of o[.][2 .. 3]
	// every weight in a low tile is zero beside what this thread's rows have seen (see above); false for NaN
	auto nothing_low_matters = [&]() {
		cp_async_wait<0>();                      // (the queries, where no tile has been computed)
		__syncthreads();
		unsigned kk = 0u;
		for (int t0 = warp; t0 < p.kt; t0 += 4 * 32) {
			const int t = t0 + 4 * lane;
			const bool low = t < p.kt && flags[t] == AP_LOW;
			unsigned *norm = p.norms + (size_t)pair * p.kt + t;
			unsigned known = low ? __ldcg(norm) : 1u;
			for (unsigned ask = __ballot_sync(0xffffffffu, known == 0u); ask; ask &= ask - 1) {
				const int who = __ffs(ask) - 1, tile = t0 + 4 * who;
				const unsigned got = ap_key_norm(k + (size_t)tile * AP_T * AP_D, min(AP_T, p.S - tile * AP_T));
				if (lane == who) __stcg(norm, known = got);
			}
			kk = max(kk, known);
		}
		unsigned *all = reinterpret_cast<unsigned *>(ap_smem);          // (the tiles are free)
		kk = __reduce_max_sync(0xffffffffu, kk);
		if (lane == 0) all[warp] = kk;
		__syncthreads();
		const float kn = sqrtf(__uint_as_float(max(max(all[0], all[1]), max(all[2], all[3]))));
		__syncthreads();
		bool ok = true;
#pragma unroll
		for (int h = 0; h < 2; ++h) {
			float qq = 0.f;
#pragma unroll
			for (int u = 0; u < 4; ++u) {
				uint32_t w[4];
				asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "r"(sq + ap_at(warp * 16 + gid + 8 * h, 4 * tig + u)) : "memory");
#pragma unroll
				for (int i = 0; i < 4; ++i) {
					const float2 e = __half22float2(*reinterpret_cast<const __half2 *>(&w[i]));
					qq = fmaf(e.x, e.x, fmaf(e.y, e.y, qq));
				}
			}
			qq += __shfl_xor_sync(0xffffffffu, qq, 1);
			qq += __shfl_xor_sync(0xffffffffu, qq, 2);
			const float most = fmaf(sqrtf(qq) * kn * 1.001f, p.scale, AP_LOW_MAX) * AP_LOG2E;          // of a low tile's scores, base 2
			ok = ok && (row + 8 * h >= p.t || mx[h] - most > 200.f);
		}
		return ok;
	};
#pragma unroll 1
	for (;;) {
		if (FULL && cur >= p.kt && any_low && !last) {
			last = true;
			if (__syncthreads_and(nothing_low_matters())) break;
			cur = next(0);
			fetch(cur, buf);
		}
		if (cur >= p.kt) break;
		const int kind = found, k0 = cur * AP_T, after = next(cur + 1);
		fetch(after, buf ^ 1);
		cp_async_wait<1>();
		__syncthreads();
		const uint32_t sk = base + buf * 2 * AP_TILE, sv = sk + AP_TILE;
		float s[8][4];
#pragma unroll
		for (int n = 0; n < 8; ++n) s[n][0] = s[n][1] = s[n][2] = s[n][3] = 0.f;
#pragma unroll
		for (int ks = 0; ks < 8; ++ks) {
			uint32_t qf[4];
			ap_ldmatrix4(qf, sq + ap_at(warp * 16 + (lane & 15), 2 * ks + (lane >> 4)));
#pragma unroll
			for (int n = 0; n < 8; n += 2) {          // 16 keys x 16 of the head's entries
				uint32_t b[4];
				ap_ldmatrix4(b, sk + ap_at(n * 8 + (lane & 7) + ((lane >> 4) << 3), 2 * ks + ((lane >> 3) & 1)));
				mma16816(s[n], qf[0], qf[1], qf[2], qf[3], b[0], b[1]);
				mma16816(s[n + 1], qf[0], qf[1], qf[2], qf[3], b[2], b[3]);
			}
		}
		uint32_t pf[4][4];                       // weights as the A operand of 16 keys each
		// scores in base 2 are s * f.  With a mask they are scaled and added to in base e, where the sum is rounded as coarsely as the softmax of a
		// row that sees large negative numbers only would have it (in base 2 half a bit more).
		const float f = kind == AP_OPEN ? p.scale * AP_LOG2E : AP_LOG2E;
		if (kind != AP_OPEN) {
			if (FULL) {
#pragma unroll
				for (int i = 0; i < 4; ++i) {
					uint32_t w[4];
					asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "r"(sm + buf * AP_MASK + i * 512) : "memory");
					const int h = i >> 1;
#pragma unroll
					for (int j = 0; j < 4; ++j) {
						const float2 add = __half22float2(*reinterpret_cast<const __half2 *>(&w[j]));
						const int n = (i & 1) * 4 + j;
						s[n][2 * h] = fmaf(s[n][2 * h], p.scale, add.x);
						s[n][2 * h + 1] = fmaf(s[n][2 * h + 1], p.scale, add.y);
					}
				}
			} else {
				const __half *m0 = mask + (long long)min(row, p.t - 1) * p.mask_st, *m1 = mask + (long long)min(row + 8, p.t - 1) * p.mask_st;
#pragma unroll
				for (int n = 0; n < 8; ++n)
#pragma unroll
					for (int j = 0; j < 2; ++j) {
						const int key = min(k0 + n * 8 + 2 * tig + j, p.S - 1);
						s[n][j] = fmaf(s[n][j], p.scale, __half2float(m0[key]));
						s[n][2 + j] = fmaf(s[n][2 + j], p.scale, __half2float(m1[key]));
					}
			}
		}
		if (k0 + AP_T > p.S) {
#pragma unroll
			for (int n = 0; n < 8; ++n)
#pragma unroll
				for (int j = 0; j < 2; ++j)
					if (k0 + n * 8 + 2 * tig + j >= p.S) s[n][j] = s[n][2 + j] = -INFINITY;
		}
		float base2[2], corr[2];
#pragma unroll
		for (int h = 0; h < 2; ++h) {
			float t = -INFINITY;
#pragma unroll
			for (int n = 0; n < 8; ++n) t = fmaxf(t, fmaxf(s[n][2 * h], s[n][2 * h + 1]));
			t = fmaxf(t, __shfl_xor_sync(0xffffffffu, t, 1));
			t = fmaxf(t, __shfl_xor_sync(0xffffffffu, t, 2));
			t = fmaxf(mx[h], t * f);
			base2[h] = t == -INFINITY ? 0.f : t;          // nothing visible so far: every weight is zero
			corr[h] = ap_exp2(mx[h] - base2[h]);
			mx[h] = t;
			sum[h] *= corr[h];
		}
#pragma unroll
		for (int n = 0; n < 16; ++n) {
			o[n][0] *= corr[0];
			o[n][1] *= corr[0];
			o[n][2] *= corr[1];
			o[n][3] *= corr[1];
		}
#pragma unroll
		for (int n = 0; n < 8; ++n) {
#pragma unroll
			for (int j = 0; j < 4; ++j) {
				s[n][j] = ap_exp2(fmaf(s[n][j], f, -base2[j >> 1]));
				sum[j >> 1] += s[n][j];
			}
			const __half2 a = __floats2half2_rn(s[n][0], s[n][1]), b = __floats2half2_rn(s[n][2], s[n][3]);
			pf[n >> 1][(n & 1) * 2] = *reinterpret_cast<const uint32_t *>(&a);
			pf[n >> 1][(n & 1) * 2 + 1] = *reinterpret_cast<const uint32_t *>(&b);
		}
#pragma unroll
		for (int ks = 0; ks < 4; ++ks)
#pragma unroll
			for (int n = 0; n < 16; n += 2) {          // 16 keys x 16 output entries
				uint32_t b[4];
				ap_ldmatrix4_trans(b, sv + ap_at(ks * 16 + (lane & 15), n + (lane >> 4)));
				mma16816(o[n], pf[ks][0], pf[ks][1], pf[ks][2], pf[ks][3], b[0], b[1]);
				mma16816(o[n + 1], pf[ks][0], pf[ks][1], pf[ks][2], pf[ks][3], b[2], b[3]);
			}
		__syncthreads();                         // the tile is free
		cur = after;
		buf ^= 1;
	}
	cp_async_wait<0>();
	__half *out = p.out + ((size_t)bi * p.t * p.heads + head) * AP_D;
#pragma unroll
	for (int h = 0; h < 2; ++h) {
		float l = sum[h];
		l += __shfl_xor_sync(0xffffffffu, l, 1);
		l += __shfl_xor_sync(0xffffffffu, l, 2);
		const float inv = l == 0.f ? 0.f : 1.f / l;          // a query that sees nothing: zeros
		if (row + 8 * h >= p.t) continue;
		__half *dst = out + (size_t)(row + 8 * h) * p.heads * AP_D + 2 * tig;
#pragma unroll
		for (int n = 0; n < 16; ++n) *reinterpret_cast<__half2 *>(dst + n * 8) = __floats2half2_rn(o[n][2 * h] * inv, o[n][2 * h + 1] * inv);
	}
}

template <typename Params>
int ap_launch(void (*kernel)(const Params), dim3 grid, int threads, size_t smem, cudaStream_t stream, const Params &p) {
	cudaLaunchConfig_t cfg = {};
	cudaLaunchAttribute attr[1];
	attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
	attr[0].val.programmaticStreamSerializationAllowed = 1;
	cfg.gridDim = grid;
	cfg.blockDim = dim3(threads);
	cfg.dynamicSmemBytes = smem;
	cfg.stream = stream;
	cfg.attrs = attr;
	cfg.numAttrs = pdl_enabled() ? 1 : 0;
	return cuda_status(cudaLaunchKernelEx(&cfg, kernel, p));
}

}   // namespace

}   // namespace gptq

using namespace gptq;

extern "C" {

size_t gptq_attn_prompt_scratch_bytes(int b, int t, int S) {
	if (b < 1 || t < 1 || S < 1) return 0;
	return (size_t)b * ((t + AP_T - 1) / AP_T) * ((S + AP_T - 1) / AP_T);
}

size_t gptq_attn_prompt_full_scratch_bytes(int mask_b, int b, int heads, int t, int S) {
	if (mask_b < 1 || b < 1 || heads < 1 || t < 1 || S < 1) return 0;
	return FullScratch(mask_b, b, heads, t, S).bytes;
}

static int prompt_shape(const void *mask, int64_t mask_sb, int64_t mask_st, int mask_b, int b, int heads, int t, int S, const void *scratch, size_t scratch_bytes) {
	if (!mask || b < 1 || heads < 1 || t < 1 || S < 1 || mask_sb < 0 || mask_st < 0 || (mask_b != 1 && mask_b != b)) return GPTQ_ERR_INVALID;
	if (b > 65535 || heads > 65535 || gptq_attn_prompt_scratch_bytes(mask_b, t, S) > (1u << 30)) return GPTQ_ERR_UNSUPPORTED;
	if (scratch && scratch_bytes < gptq_attn_prompt_scratch_bytes(mask_b, t, S)) return GPTQ_ERR_WORKSPACE;
	return GPTQ_OK;
}

int gptq_attn_prompt_prepare(const void *mask, int64_t mask_sb, int64_t mask_st, int mask_b, int b, int heads, int t, int S, const void *past_k, int64_t pk_sb, int64_t pk_sh,
							 const void *past_v, int64_t pv_sb, int64_t pv_sh, int past, void *k, void *v, void *scratch, size_t scratch_bytes, gptq_stream_t stream) {
	if (int rc = prompt_shape(mask, mask_sb, mask_st, mask_b, b, heads, t, S, scratch, scratch_bytes)) return rc;
	if (!scratch || past < 0 || past > S || (past && (!past_k || !past_v || !k || !v))) return GPTQ_ERR_INVALID;
	if (past && (!aligned16(past_k) || !aligned16(past_v) || !aligned16(k) || !aligned16(v) || ((pk_sb | pk_sh | pv_sb | pv_sh) & 7))) return GPTQ_ERR_ALIGN;
	PrepareParams p = {};
	p.mask = (const __half *)mask;
	p.mask_sb = mask_sb; p.mask_st = mask_st; p.mask_b = mask_b; p.t = t; p.S = S;
	p.qt = (t + AP_T - 1) / AP_T; p.kt = (S + AP_T - 1) / AP_T;
	p.flags = (unsigned char *)scratch;
	const FullScratch full(mask_b, b, heads, t, S);
	if (scratch_bytes >= full.bytes) {
		if (!aligned16(scratch)) return GPTQ_ERR_ALIGN;
		p.norms = reinterpret_cast<unsigned *>(p.flags + full.norms);
		p.tiles = reinterpret_cast<uint2 *>(p.flags + full.tiles);
		p.n_norms = b * heads * p.kt;
	}
	p.past_k = (const __half *)past_k; p.past_v = (const __half *)past_v;
	p.pk_sb = pk_sb; p.pk_sh = pk_sh; p.pv_sb = pv_sb; p.pv_sh = pv_sh;
	p.b = b; p.heads = heads; p.past = past;
	p.k = (__half *)k; p.v = (__half *)v;
	p.mask_ctas = mask_b * p.qt * p.kt;
	const long long units = 2ll * b * heads * past * 16;
	const int copies = (int)std::min<long long>((units + 1023) / 1024, 592);          // four units per thread, at most four CTAs per SM
	return ap_launch(attn_prepare_kernel, dim3(p.mask_ctas + copies), 256, 0, reinterpret_cast<cudaStream_t>(stream), p);
}

int gptq_attn_prompt(const void *q, int64_t q_sb, int64_t q_st, int64_t q_sh, const void *k, const void *v, const void *mask, int64_t mask_sb, int64_t mask_st, int mask_b, int b,
					 int heads, int t, int S, float scale, void *out, const void *scratch, size_t scratch_bytes, gptq_stream_t stream) {
	if (int rc = prompt_shape(mask, mask_sb, mask_st, mask_b, b, heads, t, S, scratch, scratch_bytes)) return rc;
	if (!q || !k || !v || !out || !(scale > 0.f && scale <= 3.402823466e38f)) return GPTQ_ERR_INVALID;
	if (!aligned16(q) || !aligned16(k) || !aligned16(v) || !aligned16(out) || ((q_sb | q_st | q_sh) & 7)) return GPTQ_ERR_ALIGN;
	PromptParams p = {};
	p.q = (const __half *)q; p.k = (const __half *)k; p.v = (const __half *)v; p.mask = (const __half *)mask;
	p.q_sb = q_sb; p.q_st = q_st; p.q_sh = q_sh; p.mask_sb = mask_sb; p.mask_st = mask_st; p.mask_b = mask_b;
	p.flags = (const unsigned char *)scratch;
	p.out = (__half *)out;
	p.heads = heads; p.t = t; p.S = S;
	p.qt = (t + AP_T - 1) / AP_T; p.kt = (S + AP_T - 1) / AP_T;
	p.scale = scale;
	if ((long long)p.qt * heads * b > 0x7fffffff) return GPTQ_ERR_UNSUPPORTED;          // (more output than any memory holds)
	const FullScratch full(mask_b, b, heads, t, S);
	const bool whole = scratch && scratch_bytes >= full.bytes;
	if (whole) {
		if (!aligned16(scratch)) return GPTQ_ERR_ALIGN;
		unsigned char *at = static_cast<unsigned char *>(const_cast<void *>(scratch));
		p.norms = reinterpret_cast<unsigned *>(at + full.norms);
		p.tiles = reinterpret_cast<const uint4 *>(at + full.tiles);
	}
	const int smem = 5 * AP_TILE + (whole ? 2 * AP_MASK : 0);
	const auto kernel = whole ? attn_prompt_kernel<true> : attn_prompt_kernel<false>;
	if (cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)) return cuda_status(e);
	return ap_launch(kernel, dim3(p.qt * heads * b), AP_THREADS, smem, reinterpret_cast<cudaStream_t>(stream), p);
}

}   // extern "C"
