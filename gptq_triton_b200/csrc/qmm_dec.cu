// Decode-regime (M <= 16 rows) quantised matmul on the 5th-generation tensor cores of sm_100a: every weight is read once, unpacked once
// and multiplied with all rows in one MMA.
//
// The product is computed transposed (a weight column is a lane of tensor memory, the rows of x are the N = 16 of the MMA).  The A operand
// holds the INTEGERS q - zero as fp16 (times 2^-9), which is exact; a unit of 128 K-rows lies in one group, so its fp32 sums leave tensor memory,
// are multiplied with the group's scale in fp32 and added in registers.  No weight is rounded.
//
// Split of the work: one CTA per SM (four SMs stay free, see dec_launch()), fewer when there are less than two units for each; the units of all tiles (128 columns, or 64 gate + 64 up)
// x K / 128 are one list that is cut into ranges which differ by at most one unit of 128 x 128 weights.  A CTA walks its tiles from the last to the first: the tile
// whose end lies in the next CTA's range comes first and its partial sums are handed over early, the tile whose beginning lies in the
// ranges of earlier CTAs comes last and is finished there (partial sums added in order of K: deterministic).  A CTA only ever waits for
// CTAs with lower indices.
//
//   warps 0, 3   packed weights (16 words x 128 columns); scales and zeros; into a ring of 15 units
//   warp 1       MMA issuer: eight K = 16 steps per unit; owns the tensor memory (6 stages of 64 columns of weights and of 16 columns of sums)
//   warp 2       rows of x by TMA, in the order in which they lie in memory: a pair of neighbouring nibbles is unpacked into one word
//   warps 4-7    finish every tile but the CTA's last one (hand-over or epilogue) while the next one is unpacked
//   warps 8-19   three groups of four; group j unpacks the units j, j + 3, ... and later scales and adds their sums; all of them finish the last tile
//
// What bounds it: stores to tensor memory.  A unit is 32 KB of fp16 there and takes about 0.27 us (some 64 bytes a clock; without three quarters
// of the stores, all else equal, 0.20 us a unit, which is what the weights take from HBM), and about 6 us from launch to exit (prologue, first
// copies, hand-over).  Measured against the mma.sync kernel (qmm_skinny.cuh), us, 16 rows:
//   4096 -> 4096 7.8 (11.5)   4096 -> 12288 12.2 (17.9)   11008 -> 4096 11.3 (18.4)   8192 -> 24576 29.3 (57.3)   22016 -> 8192 27.2 (55.4)
//   gate/up 4096 -> 2 x 11008 17.5 (35.3)   8192 -> 2 x 22016 50 (110)
// What brought it there (same sizes, before: 9.7, 13.8, 13.3, 31.6, 28.4, 21.6, 61): x by TMA instead of four warps that permuted it for every
// unit (gate/up 61 -> 54), the norm in a kernel of its own (82.6 -> 58), tiles finished beside the main loop and a hand-over without a
// fence per thread (4 us of each launch), stores to tensor memory in four parts that overlap with the unpacking (54 -> 50).  Eight warps per
// unit were slower (8192 -> 24576 35.4).
// On narrow layers with a deep K, where a tile is spread over many CTAs, it is the slower one; dec_min_rows() in api.cu draws the line.
// A spilled register in a loop costs an L2 round trip (shared memory takes the whole L1).
//
// Every wait is bounded; a wait that runs out sets a status word and the kernel unwinds.
#include <algorithm>
#include <atomic>

#include <cuda.h>

#include "qmm_dec.cuh"

namespace gptq {

namespace {

constexpr int DC_GROUPS = 3, DC_STAGES = 6;                  // three groups of four warps that unpack, two stages each
constexpr int DC_WORKERS = DC_GROUPS * 128, DC_FINISHERS = 128;
constexpr int DC_THREADS = 128 + DC_FINISHERS + DC_WORKERS;
constexpr int DC_W_SC = 8192, DC_W_QZ = DC_W_SC + 256, DC_W_BYTES = DC_W_QZ + 64, DC_W_STAGE = (DC_W_BYTES + 127) / 128 * 128;
constexpr int DC_W_RING = 15;                                // a multiple of the groups: a stage is always read by the same one
constexpr int DC_X_BYTES = 4096;                             // 16 rows x 128 k
constexpr int DC_RED = DC_GROUPS * 16 * 128 * 4;            // a tile's sums, one part per group; two buffers
constexpr int DC_OFF_W = DC_STAGES * DC_X_BYTES, DC_OFF_RED = DC_OFF_W + DC_W_RING * DC_W_STAGE, DC_OFF_BAR = DC_OFF_RED + 2 * DC_RED;
// mbarriers: weights and x of a unit are there; the unit has been multiplied; packed weights; a tile's sums; all MMAs
constexpr int DC_FULL = DC_OFF_BAR, DC_DONE = DC_FULL + 8 * DC_STAGES, DC_FULL_W = DC_DONE + 8 * DC_STAGES, DC_EMPTY_W = DC_FULL_W + 8 * DC_W_RING;
constexpr int DC_FULL_R = DC_EMPTY_W + 8 * DC_W_RING, DC_EMPTY_R = DC_FULL_R + 16, DC_FIN = DC_EMPTY_R + 16, DC_TMEM_ADDR = DC_FIN + 8, DC_ABORT = DC_TMEM_ADDR + 4, DC_SMEM = DC_TMEM_ADDR + 16;
constexpr int DC_A_COLS = 64, DC_STAGE_COLS = DC_A_COLS + 16, DC_TMEM_COLS = 512;
constexpr uint32_t DC_SPIN = 1u << 24;
constexpr int DC_COUNTERS = 16384;                           // bytes of the workspace's counter area; its last word is the status word
constexpr int DC_MAX_CTAS = 256, DC_SPARE = 4;
static_assert(DC_STAGES * DC_STAGE_COLS <= DC_TMEM_COLS && DC_W_RING % DC_GROUPS == 0 && DC_STAGES % DC_GROUPS == 0, "rings");
static_assert(DC_SMEM + 512 <= 227 * 1024, "shared memory per CTA");

struct DecParams {
	DecArgs a;
	int units;                   // tiles * (K / 128)
	int *flags;                  // [CTA] 1: its partial sums are there; zero between launches
	float *partial;              // [CTA][M][128]
	int *status;
	int out8;
};

// `base`: start of the CTA's shared memory
__device__ __forceinline__ bool dc_aborted(uint32_t base) {
	int f;
	asm volatile("ld.volatile.shared.s32 %0, [%1];" : "=r"(f) : "r"(base + DC_ABORT) : "memory");
	return f != 0;
}
__device__ __forceinline__ void dc_abort(uint32_t base, int *status, int code) {
	asm volatile("st.volatile.shared.s32 [%0], %1;" ::"r"(base + DC_ABORT), "r"(1) : "memory");
	atomicExch(status, code);
}
__device__ __noinline__ bool dc_wait_slow(uint32_t base, uint32_t bar, uint32_t parity) {
	return __all_sync(0xffffffffu, !dc_aborted(base) && mbar_wait_bounded(base + bar, parity, DC_SPIN));
}
__device__ __forceinline__ bool dc_wait(uint32_t base, uint32_t bar, uint32_t parity) {
	return __all_sync(0xffffffffu, mbar_try_wait(base + bar, parity)) || dc_wait_slow(base, bar, parity);
}
__device__ __forceinline__ bool dc_elect() {
	uint32_t r;
	asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xFFFFFFFF;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
	return r != 0;
}
__device__ __forceinline__ void dc_bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
	asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ uint32_t dc_lds32(uint32_t addr) {
	uint32_t r;
	asm volatile("ld.shared.u32 %0, [%1];" : "=r"(r) : "r"(addr) : "memory");
	return r;
}
__device__ __forceinline__ uint32_t dc_lds16(uint32_t addr) {
	unsigned short r;
	asm volatile("ld.shared.u16 %0, [%1];" : "=h"(r) : "r"(addr) : "memory");
	return r;
}
// Eight weights of a column, k order, as (q - zero) / 512 in fp16: exact (the nibble as a subnormal fp16 is q * 2^-24).
template <int J>
__device__ __forceinline__ uint32_t dc_pair(uint32_t e, uint32_t o, uint32_t zc) {
	uint32_t r;          // bytes: even nibble, 0, odd nibble, 0 (selectors above 7 repeat a sign bit, which is zero)
	asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(e), "r"(o), "n"(J | (8 + J) << 4 | (4 + J) << 8 | (12 + J) << 12));
	return h2_fma(r, 0x78007800u, zc);
}
__device__ __forceinline__ void dc_unpack(uint32_t w, uint32_t zc, uint32_t *out) {
	const uint32_t e = w & 0x0F0F0F0Fu, o = (w >> 4) & 0x0F0F0F0Fu;
	out[0] = dc_pair<0>(e, o, zc);
	out[1] = dc_pair<1>(e, o, zc);
	out[2] = dc_pair<2>(e, o, zc);
	out[3] = dc_pair<3>(e, o, zc);
}
__device__ __forceinline__ void dc_st16(uint32_t taddr, const uint32_t (&r)[16]) {
	asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]),
				 "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
				 : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&v)[8]) {
	uint32_t *r = reinterpret_cast<uint32_t *>(v);
	asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
				 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
				 : "r"(taddr)
				 : "memory");
}
// the NT threads that finish a tile
template <int NT>
__device__ __forceinline__ void dc_sync() { asm volatile("bar.sync %0, %1;" ::"n"(NT == DC_WORKERS ? 1 : 2), "n"(NT) : "memory"); }

// Four partial sums of `count` CTAs, `stride` floats apart, added in order of K; four CTAs' values in flight.  Out of line: its registers
// are not the main loop's.
__device__ __noinline__ float4 dec_gather(const float *src, int count, size_t stride) {
	float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
	for (int c = 0; c < count; c += 4, src += 4 * stride) {
		float4 w[4];
#pragma unroll
		for (int j = 0; j < 4; ++j)
			if (c + j < count) w[j] = __ldcg(reinterpret_cast<const float4 *>(src + j * stride));
#pragma unroll
		for (int j = 0; j < 4; ++j)
			if (c + j < count) {
				v.x += w[j].x;
				v.y += w[j].y;
				v.z += w[j].z;
				v.w += w[j].w;
			}
	}
	return v;
}

// A tile's sums of this CTA (in shared memory, one part per group): handed over to the next CTA, or finished.
template <int EPI, bool M8, int NT>
__device__ __forceinline__ void dec_finish(const DecParams &p, const float *red, int tile, int k0, bool handed_over, int wid, uint32_t base) {
	constexpr bool PAIR = (EPI == DEC_EPI_SILU);
	constexpr int TN = PAIR ? 64 : 128, ROWS = M8 ? 8 : 16;
	const DecArgs &a = p.a;
	const int lane = wid & 31, cta = blockIdx.x, np = a.K >> 7;
	auto first_unit = [&](int c) { return (int)((long long)c * p.units / (int)gridDim.x); };
	auto own = [&](int row, int col) {
		float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
		for (int g = 0; g < DC_GROUPS; ++g) {
			const float4 s = *reinterpret_cast<const float4 *>(red + (g * ROWS + row) * 128 + col);
			v.x += s.x;
			v.y += s.y;
			v.z += s.z;
			v.w += s.w;
		}
		return v;
	};
	if (handed_over) {
		// the tile goes on in the next CTA's range, which finishes it
		float4 *out = reinterpret_cast<float4 *>(p.partial + (size_t)cta * a.M * 128);
		for (int e = wid; e < a.M * 32; e += NT) __stcg(out + e, own(e >> 5, (e & 31) * 4));
		dc_sync<NT>();                              // (the release below covers what it orders)
		if (wid == 0) asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p.flags + cta), "r"(1) : "memory");
	} else {
		int c0 = cta;                               // first CTA with a share of this tile
		if (k0 > 0) {
			while (c0 > 0 && first_unit(c0) > tile * np) --c0;
			const unsigned long long t0 = global_timer_ns();
			for (int c = c0 + wid; c < cta; c += NT) {
				int f = 0;
				for (;;) {
					asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(f) : "l"(p.flags + c) : "memory");
					if (f) break;
					if (dc_aborted(base) || global_timer_ns() - t0 > 2000000000ull) {          // (bounded in time)
						dc_abort(base, p.status, 6);
						break;
					}
				}
				p.flags[c] = 0;          // clean for the next launch
			}
			dc_sync<NT>();
		}
		auto sum = [&](int row, int col) {
			const float4 s = own(row, col);
			if (c0 == cta) return s;
			const float4 v = dec_gather(p.partial + (size_t)c0 * a.M * 128 + row * 128 + col, cta - c0, (size_t)a.M * 128);
			return make_float4(v.x + s.x, v.y + s.y, v.z + s.z, v.w + s.w);
		};
		auto add4 = [](float4 &v, const __half *src) {
			v.x += __half2float(src[0]);
			v.y += __half2float(src[1]);
			v.z += __half2float(src[2]);
			v.w += __half2float(src[3]);
		};
		auto pack = [](float x, float y, float z, float w) {
			const __half2 l = __floats2half2_rn(x, y), h = __floats2half2_rn(z, w);
			return make_uint2(*reinterpret_cast<const uint32_t *>(&l), *reinterpret_cast<const uint32_t *>(&h));
		};
		const int n0 = tile * TN;
		if (EPI == DEC_EPI_PLAIN) {
			for (int e = wid; e < a.M * 32; e += NT) {          // a warp has one row
				const int row = e >> 5, col = (e & 31) * 4;
				float4 v = sum(row, col);
				if (a.bias) add4(v, a.bias + n0 + col);
				if (a.residual) add4(v, a.residual + (size_t)row * a.ldr + n0 + col);
				const uint2 o = pack(v.x, v.y, v.z, v.w);
				*reinterpret_cast<uint2 *>(a.y + (size_t)row * a.ldy + n0 + col) = o;
				if (a.ss_out) {
					const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&o.x)), g = __half22float2(*reinterpret_cast<const __half2 *>(&o.y));
					float sq = (f.x * f.x + f.y * f.y) + (g.x * g.x + g.y * g.y);
#pragma unroll
					for (int d = 4; d > 0; d >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, d);
					if ((lane & 7) == 0) a.ss_out[(size_t)row * (a.N >> 5) + tile * 4 + (lane >> 3)] = sq;
				}
			}
		} else if (EPI == DEC_EPI_SILU) {
			for (int e = wid; e < a.M * 16; e += NT) {
				const int row = e >> 4, col = (e & 15) * 4;
				const float4 v = sum(row, col), u = sum(row, col + 64);
				*reinterpret_cast<uint2 *>(a.y + (size_t)row * a.ldy + n0 + col) =
					pack(silu_f32(v.x) * u.x, silu_f32(v.y) * u.y, silu_f32(v.z) * u.z, silu_f32(v.w) * u.w);
			}
		} else {
			const int section = n0 / a.hidden, head = (n0 - section * a.hidden) >> 7;
			for (int e = wid; e < a.M * 16; e += NT) {
				const int row = e >> 4, d = (e & 15) * 4;
				int pos = a.pos[row];
				if (pos < 0 || pos >= a.max_pos) {          // never index the tables / the cache out of range
					atomicExch(p.status, 4);
					if (section != 0) continue;             // K / V of such a row are dropped, not written over cache row 0
					pos = 0;
				}
				const float4 x1 = sum(row, d), x2 = sum(row, d + 64);
				float l[4] = {x1.x, x1.y, x1.z, x1.w}, h[4] = {x2.x, x2.y, x2.z, x2.w};
				if (section < 2) {
					const __half *ct = a.cos_t + (size_t)pos * 128 + d, *st = a.sin_t + (size_t)pos * 128 + d;
#pragma unroll
					for (int j = 0; j < 4; ++j) {
						const float u = l[j], v = h[j];
						l[j] = u * __half2float(ct[j]) - v * __half2float(st[j]);
						h[j] = v * __half2float(ct[j + 64]) + u * __half2float(st[j + 64]);
					}
				}
				__half *dst;
				if (section == 0) {
					dst = a.q_out + (size_t)row * a.q_stride_m + head * 128;
				} else {
					const int bi = row / a.tokens_per_batch, ti = row - bi * a.tokens_per_batch;
					dst = (section == 1 ? a.k_out : a.v_out) + (size_t)bi * a.kv_sb + (size_t)ti * a.kv_st + (size_t)head * a.kv_sh + (size_t)pos * a.kv_sp;
				}
				if (p.out8) {
					*reinterpret_cast<uint2 *>(dst + d) = pack(l[0], l[1], l[2], l[3]);
					*reinterpret_cast<uint2 *>(dst + d + 64) = pack(h[0], h[1], h[2], h[3]);
				} else {
#pragma unroll
					for (int j = 0; j < 4; ++j) {
						dst[d + j] = __float2half_rn(l[j]);
						dst[d + 64 + j] = __float2half_rn(h[j]);
					}
				}
			}
		}
	}
}

// What a warp keeps between two tile segments.
struct DecGroup {
	int ws;                      // stage of the packed ring of its group's next unit
	uint32_t wp, ph;             // phases of that stage and of the unit's stage in tensor memory
	int st;                      // that stage
	bool ok;
};

// One group's units of a tile segment (`count` of them): unpacked into tensor memory, their sums scaled and added, the tile's sums left in
// shared memory, a part per group.  A store to tensor memory and its wait take longer than the unpacking of the words that it holds, so a
// unit is only waited for, and handed to the MMAs, when the first words of the next one have been unpacked.
template <bool PAIR, bool M8>
__device__ __forceinline__ void dec_segment(uint32_t base, uint32_t tmem, int count, DecGroup &g, float *red, uint32_t red_empty, uint32_t red_parity) {
	constexpr int ROWS = M8 ? 8 : 16;
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, grp = (warp - 8) >> 2, wt = (warp & 3) * 32 + lane;      // tensor-memory lane = weight column of the tile
	constexpr uint32_t W_ROW = PAIR ? 256 : 512;
	const uint32_t w_off = base + DC_OFF_W + (PAIR ? (uint32_t)((wt >> 6) * 4096 + (wt & 63) * 4) : (uint32_t)(wt * 4));
	const uint32_t sc_off = base + DC_OFF_W + DC_W_SC + wt * 2, qz_off = base + DC_OFF_W + DC_W_QZ + (wt >> 3) * 4;
	const uint32_t ta = tmem + ((uint32_t)((warp & 3) * 32) << 16);
	float acc[ROWS];
#pragma unroll
	for (int r = 0; r < ROWS; ++r) acc[r] = 0.f;
	float sc0 = 0.f, sc1 = 0.f, sc2 = 0.f;          // scales of the unit in hand and of the two before
	uint32_t zc = 0, w[16];
	auto fetch = [&]() {
		const uint32_t o = g.ws * DC_W_STAGE;
		g.ok = g.ok && dc_wait(base, DC_FULL_W + 8 * g.ws, g.wp);
		if (!g.ok) return;
#pragma unroll
		for (int r = 0; r < 16; ++r) w[r] = dc_lds32(w_off + o + r * W_ROW);
		sc0 = 512.f * __half2float(__ushort_as_half((unsigned short)dc_lds16(sc_off + o)));
		const uint32_t zz = ((dc_lds32(qz_off + o) >> ((wt & 7) * 4)) & 0xFu) + 1u;
		zc = h2_mul(h2_sub((0x6400u + zz) * 0x00010001u, MAGIC_1024), 0x98009800u);      // half2(-zero / 512)
	};
	auto other = [&](int st) { return st >= DC_GROUPS ? st - DC_GROUPS : st + DC_GROUPS; };
	auto hand_over = [&](int st) {                  // a unit's weights have landed
		tmem_st_wait();
		tc_fence_before();
		__syncwarp();
		if (lane == 0) mbar_arrive(base + DC_FULL + 8 * st);
	};
	auto add = [&](int st, float scale) {           // a stage's sums: tensor memory -> registers
#pragma unroll
		for (int h = 0; h < ROWS; h += 8) {
			float d[8];
			tmem_ld8(ta + st * DC_STAGE_COLS + DC_A_COLS + h, d);
			tmem_ld_wait();
#pragma unroll
			for (int r = 0; r < 8; ++r) {
				asm volatile("" : "+f"(d[r]));              // not before the wait
				acc[h + r] = fmaf(scale, d[r], acc[h + r]);
			}
		}
	};
	if (count > 0) fetch();
#pragma unroll 1
	for (int i = 0; i < count && g.ok; ++i) {
		uint32_t o[16];
#pragma unroll
		for (int r = 0; r < 4; ++r) dc_unpack(w[r], zc, o + 4 * r);
		if (i > 0) hand_over(other(g.st));
		g.ok = dc_wait(base, DC_DONE + 8 * g.st, g.ph ^ 1);          // the unit that used this stage has been multiplied
		if (!g.ok) break;
		tc_fence_after();
		const uint32_t at = ta + g.st * DC_STAGE_COLS;
		dc_st16(at, o);
#pragma unroll
		for (int b = 1; b < 4; ++b) {
			uint32_t v[16];
#pragma unroll
			for (int r = 0; r < 4; ++r) dc_unpack(w[4 * b + r], zc, v + 4 * r);
			dc_st16(at + 16 * b, v);
		}
		__syncwarp();
		if (lane == 0) mbar_arrive(base + DC_EMPTY_W + 8 * g.ws);
		g.ws += DC_GROUPS;
		if (g.ws >= DC_W_RING) {
			g.ws -= DC_W_RING;
			g.wp ^= 1;
		}
		if (i >= 2) add(g.st, sc2);                 // (an earlier segment's sums have been read)
		sc2 = sc1;
		sc1 = sc0;
		if (i + 1 < count) fetch();
		g.st += DC_GROUPS;
		if (g.st >= DC_STAGES) {
			g.st -= DC_STAGES;
			g.ph ^= 1;
		}
	}
	if (g.ok && count > 0) {
		// the last two units: the next one's stage holds the older of them
		hand_over(other(g.st));
		if (count > 1) {
			g.ok = dc_wait(base, DC_DONE + 8 * g.st, g.ph ^ 1);
			tc_fence_after();
			if (g.ok) add(g.st, sc2);
		}
		g.ok = g.ok && dc_wait(base, DC_DONE + 8 * other(g.st), g.st >= DC_GROUPS ? g.ph : g.ph ^ 1);
		tc_fence_after();
		if (g.ok) add(other(g.st), sc1);
	}
	tc_fence_before();
	g.ok = g.ok && dc_wait(base, red_empty, red_parity);          // the tile two segments back has left the buffer
#pragma unroll
	for (int r = 0; r < ROWS; ++r) red[(grp * ROWS + r) * 128 + wt] = acc[r];
}

template <int EPI, bool M8>
__global__ void __launch_bounds__(DC_THREADS, 1) dec_kernel(const __grid_constant__ CUtensorMap tmw0, const __grid_constant__ CUtensorMap tmw1,
															const __grid_constant__ CUtensorMap tmx, const __grid_constant__ DecParams p) {
	extern __shared__ __align__(1024) unsigned char smem[];
	constexpr bool PAIR = (EPI == DEC_EPI_SILU);             // 64 gate and 64 up columns per tile
	constexpr int TN = PAIR ? 64 : 128;
	const DecArgs &a = p.a;
	const int tid = threadIdx.x, warp = tid >> 5, cta = blockIdx.x;
	const int np = a.K >> 7;
	auto first_unit = [&](int c) { return (int)((long long)c * p.units / (int)gridDim.x); };
	const int lo = first_unit(cta), hi = first_unit(cta + 1), n = hi - lo;
	const uint32_t base = smem_u32(smem);

	if (tid == 0) {
		for (int s = 0; s < DC_STAGES; ++s) {
			mbar_init(base + DC_FULL + 8 * s, 5);             // four warps that unpack, rows of x
			mbar_init(base + DC_DONE + 8 * s, 1);             // sums are there, A and B are free
		}
		for (int s = 0; s < DC_W_RING; ++s) {
			mbar_init(base + DC_FULL_W + 8 * s, 2);           // words; scales and zeros
			mbar_init(base + DC_EMPTY_W + 8 * s, 4);
		}
		for (int s = 0; s < 2; ++s) {
			mbar_init(base + DC_FULL_R + 8 * s, DC_WORKERS / 32);
			mbar_init(base + DC_EMPTY_R + 8 * s, DC_FINISHERS / 32);
		}
		mbar_init(base + DC_FIN, 1);
		*reinterpret_cast<volatile int *>(smem + DC_ABORT) = 0;
		fence_mbar_init();
		tma_prefetch_desc(&tmw0);
		if (PAIR) tma_prefetch_desc(&tmw1);
		tma_prefetch_desc(&tmx);
	}
	if (warp == 1) {
		tmem_alloc(base + DC_TMEM_ADDR, DC_TMEM_COLS);
		tmem_relinquish();
	}
	tc_fence_before();
	__syncthreads();
	tc_fence_after();
	const uint32_t tmem = *reinterpret_cast<uint32_t *>(smem + DC_TMEM_ADDR);

	if (warp == 0 || warp == 3) {
		// ---------------- packed weights (warp 0), scales and zeros (warp 3); they depend on no earlier kernel ----------------
		// Two warps, and nothing but additions per unit: with one warp and a division the chain of these instructions was the bound.
		const int nz = a.N >> 3, gk = a.groupsize >> 7;
		int s = 0, tile = (hi - 1) / np, left = n;
		uint32_t ph = 1, dst = base + DC_OFF_W, bar = DC_FULL_W;
		const bool one = dc_elect();
		bool ok = true;
		while (left > 0 && ok) {
			const int k0 = max(lo - tile * np, 0), len = min(hi - tile * np, np) - k0, n0 = tile * TN, g0 = k0 / gk;
			int in_group = gk - (k0 - g0 * gk), row = k0 * 16;
			size_t so = (size_t)g0 * a.N + n0, zo = (size_t)g0 * nz + (n0 >> 3);
			const __half *sc0 = a.sc0 + so, *sc1 = PAIR ? a.sc1 + so : nullptr;
			const int32_t *qz0 = a.qz0 + zo, *qz1 = PAIR ? a.qz1 + zo : nullptr;
			left -= len;
			--tile;
			for (int i = 0; i < len; ++i) {
				ok = dc_wait(base, bar + (DC_EMPTY_W - DC_FULL_W), ph);
				if (!ok) break;
				if (one) {
					if (warp == 0) {
						mbar_arrive_expect_tx(base + bar, DC_W_SC);
						tma_load_2d(dst, &tmw0, n0, row, base + bar);
						if (PAIR) tma_load_2d(dst + 4096, &tmw1, n0, row, base + bar);
					} else {
						mbar_arrive_expect_tx(base + bar, DC_W_BYTES - DC_W_SC);
						dc_bulk_load(dst + DC_W_SC, sc0, TN * 2, base + bar);
						dc_bulk_load(dst + DC_W_QZ, qz0, TN / 2, base + bar);
						if (PAIR) {
							dc_bulk_load(dst + DC_W_SC + 128, sc1, TN * 2, base + bar);
							dc_bulk_load(dst + DC_W_QZ + 32, qz1, TN / 2, base + bar);
						}
					}
				}
				__syncwarp();
				row += 16;
				if (--in_group == 0) {
					in_group = gk;
					sc0 += a.N;
					qz0 += nz;
					if (PAIR) {
						sc1 += a.N;
						qz1 += nz;
					}
				}
				dst += DC_W_STAGE;
				bar += 8;
				if (++s == DC_W_RING) {
					s = 0;
					dst = base + DC_OFF_W;
					bar = DC_FULL_W;
					ph ^= 1;
				}
			}
		}
		if (!ok) {
			dc_abort(base, p.status, 1);
			const unsigned long long t0 = global_timer_ns();          // copies in flight land before the CTA may end
			while (global_timer_ns() - t0 < 1000000ull) __nanosleep(1000);
		}
	} else if (warp == 2) {
		// ---------------- rows of x: 16 rows x 128 k per unit, rows that do not exist are filled with zeros ----------------
		const bool one = dc_elect();
		pdl_wait();
		// behind the wait: what ran before this kernel is complete when its successor starts; not at all when it stores several cache rows of a
		// sequence (see common.cuh)
		if (EPI != DEC_EPI_ROPE || a.tokens_per_batch == 1) pdl_trigger();
		int s = 0, tile = (hi - 1) / np, left = n;
		uint32_t ph = 1;
		bool ok = true;
		while (left > 0 && ok) {
			const int k0 = max(lo - tile * np, 0), len = min(hi - tile * np, np) - k0;
			left -= len;
			--tile;
			for (int k = k0 * 128; k < (k0 + len) * 128; k += 128) {
				ok = dc_wait(base, DC_DONE + 8 * s, ph);
				if (!ok) break;
				if (one) {
					const uint32_t bar = base + DC_FULL + 8 * s, dst = base + s * DC_X_BYTES;
					mbar_arrive_expect_tx(bar, DC_X_BYTES);
					tma_load_2d(dst, &tmx, k, 0, bar);
					tma_load_2d(dst + DC_X_BYTES / 2, &tmx, k + 64, 0, bar);
				}
				__syncwarp();
				if (++s == DC_STAGES) {
					s = 0;
					ph ^= 1;
				}
			}
		}
		if (!ok) {
			dc_abort(base, p.status, 1);
			const unsigned long long t0 = global_timer_ns();
			while (global_timer_ns() - t0 < 1000000ull) __nanosleep(1000);
		}
	} else if (warp == 1) {
		// ---------------- MMA issuer: eight K = 16 steps per unit ----------------
		const uint32_t idesc = (1u << 4) | ((uint32_t)(16 >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);   // D fp32, A/B fp16 K-major, N = 16, M = 128
		const uint64_t xd = smem_desc_sw128(base);
		uint32_t ph = 0;
		int s = 0;
		const bool one = dc_elect();
		bool ok = true;
		for (int i = 0; i < n; ++i) {
			ok = dc_wait(base, DC_FULL + 8 * s, ph);
			if (!ok) break;
			tc_fence_after();
			if (one) {
				const uint32_t at = tmem + s * DC_STAGE_COLS, d = at + DC_A_COLS;
				const uint64_t xs = xd + (uint64_t)(s * (DC_X_BYTES >> 4));
#pragma unroll
				for (int k = 0; k < 8; ++k) umma_f16_ts(d, at + 8 * k, xs + (uint64_t)((k >> 2) * 128 + 2 * (k & 3)), idesc, k ? 1u : 0u);
				umma_commit(base + DC_DONE + 8 * s);
			}
			__syncwarp();
			if (++s == DC_STAGES) {
				s = 0;
				ph ^= 1;
			}
		}
		if (!ok) dc_abort(base, p.status, 3);
		if (one) umma_commit(base + DC_FIN);
		__syncwarp();
	} else if (warp < 8) {
		// ---------------- finish every tile segment but the last one, while the next is unpacked ----------------
		float *red = reinterpret_cast<float *>(smem + DC_OFF_RED);
		int tile = (hi - 1) / np, b = 0;
		uint32_t ph = 0;
		pdl_wait();                                         // outputs, residual and the exchange area belong to earlier kernels until here
		for (; tile * np > lo; --tile) {
			if (!dc_wait(base, DC_FULL_R + 8 * b, ph)) break;
			dec_finish<EPI, M8, DC_FINISHERS>(p, red + b * (DC_RED / 4), tile, 0, hi < (tile + 1) * np, tid - 128, base);
			dc_sync<DC_FINISHERS>();
			if ((tid & 31) == 0) mbar_arrive(base + DC_EMPTY_R + 8 * b);
			b ^= 1;
			ph ^= b == 0;
		}
	} else {
		// ---------------- unpack, scale and add; finish the last segment ----------------
		float *red = reinterpret_cast<float *>(smem + DC_OFF_RED);
		int tile = (hi - 1) / np, end = 0, next = (warp - 8) >> 2, b = 0;      // units of the segments so far; next unit of this warp's group
		uint32_t ph = 1;
		DecGroup g = {next, 0u, 0u, next, true};
		for (;; --tile) {
			const int k0 = max(lo - tile * np, 0), k1 = min(hi - tile * np, np);
			end += k1 - k0;
			const int count = max(0, (end - next + DC_GROUPS - 1) / DC_GROUPS);
			dec_segment<PAIR, M8>(base, tmem, count, g, red + b * (DC_RED / 4), DC_EMPTY_R + 8 * b, ph);
			next += DC_GROUPS * count;
			if (!g.ok) dc_abort(base, p.status, 3);
			if (end >= n) {
				pdl_wait();
				dc_sync<DC_WORKERS>();
				dec_finish<EPI, M8, DC_WORKERS>(p, red + b * (DC_RED / 4), tile, k0, k1 < np, tid - 256, base);
				break;
			}
			__syncwarp();
			if ((tid & 31) == 0) mbar_arrive(base + DC_FULL_R + 8 * b);
			b ^= 1;
			ph ^= b == 0;
		}
	}
	tc_fence_before();
	__syncthreads();
	if (warp == 1) {
		// tensor memory goes back only after every MMA issued above has completed (also when unwinding)
		if ((tid & 31) == 0) mbar_wait_bounded(base + DC_FIN, 0, DC_SPIN);
		__syncwarp();
		tc_fence_after();
		tmem_dealloc(tmem, DC_TMEM_COLS);
	}
}

}   // namespace

EncodeTiledFn tensor_map_encoder();      // defined in api.cu
bool pdl_enabled();

bool dec_shape_ok(int M, int K, int N, int groupsize) {
	return M >= 1 && M <= 16 && N % 128 == 0 && K % 128 == 0 && groupsize % 128 == 0 && K % groupsize == 0 && (long long)(N / 64) * (K / 128) < (1 << 24);
}
size_t dec_ws_bytes(int M) { return DC_COUNTERS + (size_t)DC_MAX_CTAS * std::min(std::max(M, 0), 16) * 128 * sizeof(float); }

static int dec_map(const int32_t *qw, int K, int N, int cols, CUtensorMap *out) {
	EncodeTiledFn enc = tensor_map_encoder();
	if (!enc) return GPTQ_ERR_CUDA;
	cuuint64_t dims[2] = {(cuuint64_t)N, (cuuint64_t)(K / 8)}, strides[1] = {(cuuint64_t)N * 4};
	cuuint32_t box[2] = {(cuuint32_t)cols, 16}, estr[2] = {1, 1};
	CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_INT32, 2, const_cast<int32_t *>(qw), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
					 CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
	if (r != CUDA_SUCCESS) {
		g_last_cuda_error = (int)r;
		return GPTQ_ERR_CUDA;
	}
	return GPTQ_OK;
}

// fp16 rows of x, boxes of 64 k x 16 rows, 128-byte swizzle
static int dec_map_x(const DecArgs &a, CUtensorMap *out) {
	cuuint64_t dims[2] = {(cuuint64_t)a.K, (cuuint64_t)a.M}, strides[1] = {(cuuint64_t)a.ldx * 2};
	cuuint32_t box[2] = {64, 16}, estr[2] = {1, 1};
	CUresult r = tensor_map_encoder()(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<__half *>(a.x), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
									  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
	if (r != CUDA_SUCCESS) {
		g_last_cuda_error = (int)r;
		return GPTQ_ERR_CUDA;
	}
	return GPTQ_OK;
}

template <int EPI, bool M8>
static int dec_go(const DecParams &p, int grid, int dev, cudaStream_t stream) {
	constexpr int TN = EPI == DEC_EPI_SILU ? 64 : 128;
	auto k = dec_kernel<EPI, M8>;
	static std::atomic<bool> ready[64];
	if (!ready[dev]) {
		cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, DC_SMEM);
		if (e != cudaSuccess) return cuda_status(e);
		ready[dev] = true;
	}
	alignas(64) CUtensorMap tmw0, tmw1, tmx;
	if (int rc = dec_map(p.a.qw0, p.a.K, p.a.N, TN, &tmw0)) return rc;
	tmw1 = tmw0;
	if (EPI == DEC_EPI_SILU)
		if (int rc = dec_map(p.a.qw1, p.a.K, p.a.N, TN, &tmw1)) return rc;
	if (int rc = dec_map_x(p.a, &tmx)) return rc;
	cudaLaunchConfig_t cfg = {};
	cudaLaunchAttribute attr[1];
	attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
	attr[0].val.programmaticStreamSerializationAllowed = 1;
	cfg.gridDim = dim3(grid);
	cfg.blockDim = dim3(DC_THREADS);
	cfg.dynamicSmemBytes = DC_SMEM;
	cfg.stream = stream;
	cfg.attrs = attr;
	cfg.numAttrs = pdl_enabled() ? 1 : 0;
	return cuda_status(cudaLaunchKernelEx(&cfg, k, tmw0, tmw1, tmx, p));
}

int dec_launch(const DecArgs &a, int epi, void *workspace, size_t ws_bytes, cudaStream_t stream) {
	if (!workspace || ws_bytes < dec_ws_bytes(a.M)) return GPTQ_ERR_WORKSPACE;
	int dev = 0, sms = 0;
	if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return GPTQ_ERR_CUDA;
	if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 148;
	DecParams p = {};
	p.a = a;
	p.units = a.N / (epi == DEC_EPI_SILU ? 64 : 128) * (a.K / 128);
	p.flags = reinterpret_cast<int *>(workspace);
	p.status = p.flags + DC_COUNTERS / 4 - 1;
	p.partial = reinterpret_cast<float *>(reinterpret_cast<unsigned char *>(workspace) + DC_COUNTERS);
	auto even = [](const void *ptr) { return (reinterpret_cast<uintptr_t>(ptr) & 7u) == 0; };
	p.out8 = even(a.q_out) && even(a.k_out) && even(a.v_out) && ((a.q_stride_m | a.kv_sb | a.kv_st | a.kv_sh | a.kv_sp) & 3) == 0;
	// At least two units per CTA, and four SMs left free: a CTA needs a whole SM, so with one on each SM the next launch's CTA starts only when the
	// last one of this launch has left its SM, and the launch lasts as long as that one needs from its start (8.7 us where the others are done 5.3 us
	// after their wait).  With SMs to spare every CTA of the next launch fills its ring beforehand.  148 / 147 / 144 / 140 CTAs, 16 rows, us:
	// 4096 -> 4096 8.4 / 8.2 / 7.8 / 7.8, 4096 -> 12288 12.7 / 12.6 / 12.2 / 12.4, 8192 -> 24576 (83 units for each) 29.8 / 29.4 / 29.3 / 30.3; a decode
	// step of 4 layers of 4096 355 -> 342.  From 100 units on the lost SMs weigh more: gate/up of 8192 -> 2 x 22016 (149 units) 50.1 / 50.2 / 50.8 / 51.8.
	const int spare = sms > DC_SPARE && p.units < 100 * sms ? DC_SPARE : 0;
	const int grid = std::max(1, std::min({sms - spare, DC_MAX_CTAS, p.units / 2}));
	const bool m8 = a.M <= 8;
	switch (epi) {
		case DEC_EPI_PLAIN: return m8 ? dec_go<DEC_EPI_PLAIN, true>(p, grid, dev, stream) : dec_go<DEC_EPI_PLAIN, false>(p, grid, dev, stream);
		case DEC_EPI_SILU: return m8 ? dec_go<DEC_EPI_SILU, true>(p, grid, dev, stream) : dec_go<DEC_EPI_SILU, false>(p, grid, dev, stream);
		case DEC_EPI_ROPE: return m8 ? dec_go<DEC_EPI_ROPE, true>(p, grid, dev, stream) : dec_go<DEC_EPI_ROPE, false>(p, grid, dev, stream);
	}
	return GPTQ_ERR_INVALID;
}

}   // namespace gptq
