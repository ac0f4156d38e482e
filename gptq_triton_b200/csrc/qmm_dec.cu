// Decode-regime (M <= 16 rows) quantised matmul on the 5th-generation tensor cores of sm_100a: every weight is read once, unpacked once
// and multiplied with all rows in one MMA.
//
// The product is computed transposed (a weight column is a lane of tensor memory, the rows of x are the N = 16 of the MMA).  The A operand
// holds the INTEGERS q - zero as fp16, which is exact; a unit of 128 K-rows lies in one group, so its fp32 sums leave tensor memory, are
// multiplied with the group's scale in fp32 and added in registers.  No weight is rounded.
//
// Split of the work: one CTA per SM, fewer when there are less than two units for each; the units of all tiles (128 columns, or 64 gate + 64 up)
// x K / 128 are one list that is cut into ranges which differ by at most one unit of 128 x 128 weights.  A CTA walks its tiles from the last to the first: the tile
// whose end lies in the next CTA's range comes first and its partial sums are handed over early, the tile whose beginning lies in the
// ranges of earlier CTAs comes last and is finished there (partial sums added in order of K: deterministic).  A CTA only ever waits for
// CTAs with lower indices.
//
//   warps 0, 3   packed weights (16 words x 128 columns); scales and zeros; into a ring of 18 units
//   warp 1       MMA issuer: eight K = 16 steps per unit
//   warp 2       owns the tensor memory (6 stages of 64 columns of weights and of 16 columns of sums)
//   warps 4-7    rows of x, a warp per unit in turn: RMSNorm factor where asked for, k order 0 4 1 5 2 6 3 7 of each eight (as the nibbles of a word unpack in
//                pairs), into the 128-byte-swizzled B operand
//   warps 8-19   three groups of four; group j unpacks the units j, j + 3, ... and later scales and adds their sums
//
// What bounds it: the instructions around a unit (0.21 - 0.25 us per unit and CTA, 3.2 - 3.7 TB/s of weights at 90 MB and more) and about
// 8 us from launch to exit (prologue, first copies, hand-over).  Measured against the mma.sync kernel (qmm_skinny.cuh), us, 16 rows:
//   4096 -> 4096 10.3 (11.7)   4096 -> 12288 14.4 (18.0)   11008 -> 4096 13.5 (18.3)   8192 -> 24576 32.0 (57.1)   22016 -> 8192 28.6 (55.6)
//   gate/up 4096 -> 2 x 11008 21.8 (34.8)   8192 -> 2 x 22016 61 (110)
// On narrow layers with a deep K, where a tile is spread over many CTAs, it is the slower one; dec_min_rows() in api.cu draws the line.
// A spilled register in a loop costs an L2 round trip (shared memory takes the whole L1): with spills the last line read 154 us.
//
// Every wait is bounded; a wait that runs out sets a status word and the kernel unwinds.
#include <algorithm>
#include <atomic>

#include <cuda.h>

#include "qmm_dec.cuh"

namespace gptq {

namespace {

constexpr int DC_GROUPS = 3, DC_STAGES = 6;                  // two stages per group
constexpr int DC_WORKERS = DC_GROUPS * 128;
constexpr int DC_THREADS = 256 + DC_WORKERS;
constexpr int DC_W_SC = 8192, DC_W_QZ = DC_W_SC + 256, DC_W_BYTES = DC_W_QZ + 64, DC_W_STAGE = (DC_W_BYTES + 127) / 128 * 128;
constexpr int DC_W_RING = 18;                                // a multiple of the groups: a stage is always read by the same one
constexpr int DC_X_STAGE = 4096;                             // 16 rows x 128 k
constexpr int DC_RED = DC_GROUPS * 16 * 128 * 4;
constexpr int DC_OFF_W = DC_STAGES * DC_X_STAGE, DC_OFF_RED = DC_OFF_W + DC_W_RING * DC_W_STAGE, DC_OFF_BAR = DC_OFF_RED + DC_RED;
constexpr int DC_SMEM = DC_OFF_BAR + (2 * DC_STAGES + 2 * DC_W_RING + 1) * 8 + 16;
constexpr int DC_D_COLS = 16, DC_TMEM_COLS = 512;
constexpr uint32_t DC_SPIN = 1u << 24;
constexpr int DC_COUNTERS = 16384;                           // bytes of the workspace's counter area; its last word is the status word
constexpr int DC_MAX_CTAS = 256;
static_assert(DC_STAGES * (64 + DC_D_COLS) <= DC_TMEM_COLS && DC_W_RING % DC_GROUPS == 0 && DC_STAGES == 2 * DC_GROUPS, "rings");
static_assert(DC_SMEM + 512 <= 227 * 1024, "shared memory per CTA");

struct DecParams {
	DecArgs a;
	int units;                   // tiles * (K / 128)
	int *flags;                  // [CTA] 1: its partial sums are there; zero between launches
	float *partial;              // [CTA][M][128]
	int *status;
	int out8;
};

__device__ __noinline__ bool dc_wait_slow(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
	return __all_sync(0xffffffffu, !*abort_flag && mbar_wait_bounded(bar, parity, DC_SPIN));
}
__device__ __forceinline__ bool dc_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
	return __all_sync(0xffffffffu, mbar_try_wait(bar, parity)) || dc_wait_slow(bar, parity, abort_flag);
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
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&v)[8]) {
	uint32_t *r = reinterpret_cast<uint32_t *>(v);
	asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
				 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
				 : "r"(taddr)
				 : "memory");
}
__device__ __forceinline__ void dc_workers_sync() { asm volatile("bar.sync 1, %0;" ::"n"(DC_WORKERS) : "memory"); }

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
template <int EPI, bool M8>
__device__ __forceinline__ void dec_finish(const DecParams &p, const float *red, int tile, int k0, bool handed_over, int wid, volatile int *s_abort) {
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
		for (int e = wid; e < a.M * 32; e += DC_WORKERS) __stcg(out + e, own(e >> 5, (e & 31) * 4));
		__threadfence();
		dc_workers_sync();
		if (wid == 0) asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p.flags + cta), "r"(1) : "memory");
	} else {
		int c0 = cta;                               // first CTA with a share of this tile
		if (k0 > 0) {
			while (c0 > 0 && first_unit(c0) > tile * np) --c0;
			const unsigned long long t0 = global_timer_ns();
			for (int c = c0 + wid; c < cta; c += DC_WORKERS) {
				int f = 0;
				for (;;) {
					asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(f) : "l"(p.flags + c) : "memory");
					if (f) break;
					if (*s_abort || global_timer_ns() - t0 > 2000000000ull) {          // (bounded in time)
						*s_abort = 1;
						atomicExch(p.status, 6);
						break;
					}
				}
				p.flags[c] = 0;          // clean for the next launch
			}
			dc_workers_sync();
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
			for (int e = wid; e < a.M * 32; e += DC_WORKERS) {          // a warp has one row
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
			for (int e = wid; e < a.M * 16; e += DC_WORKERS) {
				const int row = e >> 4, col = (e & 15) * 4;
				const float4 v = sum(row, col), u = sum(row, col + 64);
				*reinterpret_cast<uint2 *>(a.y + (size_t)row * a.ldy + n0 + col) =
					pack(silu_f32(v.x) * u.x, silu_f32(v.y) * u.y, silu_f32(v.z) * u.z, silu_f32(v.w) * u.w);
			}
		} else {
			const int section = n0 / a.hidden, head = (n0 - section * a.hidden) >> 7;
			for (int e = wid; e < a.M * 16; e += DC_WORKERS) {
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

// x: warp xw stages the units xw, xw + 4, ...; lane -> eight k of every other row.  Out of line like the epilogue: a spilled register in
// a loop costs an L2 round trip here (shared memory takes all of the L1).
template <int EPI, bool M8>
__device__ __noinline__ void dec_stage_x(const DecParams &p, int xw, int lane, uint32_t sX, uint32_t bar_full, uint32_t bar_done, float *s_inv, volatile int *s_abort) {
	constexpr int ROWS = M8 ? 8 : 16;
	const DecArgs &a = p.a;
	const int np = a.K >> 7;
	auto first_unit = [&](int c) { return (int)((long long)c * p.units / (int)gridDim.x); };
	const int lo = first_unit(blockIdx.x), hi = first_unit(blockIdx.x + 1), n = hi - lo;
	auto fail = [&](int code) {
		*s_abort = 1;
		atomicExch(p.status, code);
	};
	const int u = lane & 15, r0 = lane >> 4;
	pdl_wait();
	// behind the wait: what ran before this kernel is complete when its successor starts; not at all when it stores several cache rows of a
	// sequence (see common.cuh)
	if (EPI != DEC_EPI_ROPE || a.tokens_per_batch == 1) pdl_trigger();
	const bool rms = EPI != DEC_EPI_PLAIN && a.rms_w != nullptr;
	if (rms) {
		// 1 / rms of every row from the per-tile sums the producing kernel left (fixed order)
		for (int r = xw; r < a.M; r += 4) {
			float v = 0.f;
			for (int i = lane; i < a.ss_tiles; i += 32) v += __ldcg(a.ss_in + (size_t)r * a.ss_tiles + i);
#pragma unroll
			for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
			if (lane == 0) s_inv[r] = rsqrtf(v / (float)a.K + a.rms_eps);
		}
		asm volatile("bar.sync 2, 128;" ::: "memory");
	}
	constexpr int H = ROWS / 2;
	const __half *src = a.x + (size_t)r0 * a.ldx + u * 8;
	const size_t step = (size_t)2 * a.ldx;
	uint4 v[H], wq;
	int tile = (hi - 1) / np, k0 = max(lo - tile * np, 0), begin = 0, end = min(hi - tile * np, np) - k0;
	auto load = [&](int i) {
		while (i >= end) {                              // the segment that holds unit i
			--tile;
			k0 = max(lo - tile * np, 0);
			begin = end;
			end += np - k0;
		}
		const int k = (k0 + i - begin) * 128;
#pragma unroll
		for (int h = 0; h < H; ++h)
			if (r0 + 2 * h < a.M) v[h] = __ldcg(reinterpret_cast<const uint4 *>(src + h * step + k));
		if (rms) wq = __ldg(reinterpret_cast<const uint4 *>(a.rms_w + k + u * 8));
	};
	if (xw < n) load(xw);
	int s = xw;
	uint32_t ph = 1;
	for (int i = xw; i < n; i += 4) {
		if (!dc_wait(bar_done + 8 * s, ph, s_abort)) { fail(3); break; }
		const uint32_t dst = sX + s * DC_X_STAGE + (u >> 3) * 2048;
#pragma unroll
		for (int h = 0; h < H; ++h) {
			const int row = r0 + 2 * h;
			if (row < a.M) {
				uint4 x = v[h];
				if (rms) {
					// x * inv_rms * w: fp32 product, one fp16 rounding (same expression as rmsnorm_kernel)
					const float inv = s_inv[row];
					const uint32_t xv[4] = {x.x, x.y, x.z, x.w}, wv[4] = {wq.x, wq.y, wq.z, wq.w};
					uint32_t ov[4];
#pragma unroll
					for (int e = 0; e < 4; ++e) {
						const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&xv[e])), g = __half22float2(*reinterpret_cast<const __half2 *>(&wv[e]));
						const __half2 o = __floats2half2_rn(f.x * inv * g.x, f.y * inv * g.y);
						ov[e] = *reinterpret_cast<const uint32_t *>(&o);
					}
					x = make_uint4(ov[0], ov[1], ov[2], ov[3]);
				}
				const uint32_t at = dst + (row >> 3) * 1024 + (row & 7) * 128 + (((u & 7) ^ (row & 7)) << 4);
				asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(at), "r"(__byte_perm(x.x, x.z, 0x5410)), "r"(__byte_perm(x.x, x.z, 0x7632)),
							 "r"(__byte_perm(x.y, x.w, 0x5410)), "r"(__byte_perm(x.y, x.w, 0x7632))
							 : "memory");
			}
		}
		fence_proxy_async();                            // (no load of this warp is in flight that it would wait for)
		__syncwarp();
		if (lane == 0) mbar_arrive(bar_full + 8 * s);
		if (i + 4 < n) load(i + 4);
		s += 4;
		if (s >= DC_STAGES) {
			s -= DC_STAGES;
			ph ^= 1;
		}
	}
	__syncwarp();
}

template <int EPI, bool M8>
__global__ void __launch_bounds__(DC_THREADS, 1) dec_kernel(const __grid_constant__ CUtensorMap tmw0, const __grid_constant__ CUtensorMap tmw1,
															const __grid_constant__ DecParams p) {
	extern __shared__ __align__(1024) unsigned char smem[];
	__shared__ float s_inv[16];
	constexpr bool PAIR = (EPI == DEC_EPI_SILU);             // 64 gate and 64 up columns per tile
	constexpr int TN = PAIR ? 64 : 128, ROWS = M8 ? 8 : 16;
	const DecArgs &a = p.a;
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, cta = blockIdx.x;
	const int np = a.K >> 7;
	auto first_unit = [&](int c) { return (int)((long long)c * p.units / (int)gridDim.x); };
	const int lo = first_unit(cta), hi = first_unit(cta + 1), n = hi - lo;

	const uint32_t sX = smem_u32(smem), sW = sX + DC_OFF_W;
	float *red = reinterpret_cast<float *>(smem + DC_OFF_RED);
	uint64_t *bars = reinterpret_cast<uint64_t *>(smem + DC_OFF_BAR);
	const uint32_t bar_full = smem_u32(bars), bar_done = bar_full + 8 * DC_STAGES, bar_full_w = bar_done + 8 * DC_STAGES, bar_empty_w = bar_full_w + 8 * DC_W_RING;
	const uint32_t bar_fin = bar_empty_w + 8 * DC_W_RING;
	uint32_t *s_tmem = reinterpret_cast<uint32_t *>(bars + 2 * DC_STAGES + 2 * DC_W_RING + 1);
	volatile int *s_abort = reinterpret_cast<volatile int *>(s_tmem + 1);

	if (tid == 0) {
		for (int s = 0; s < DC_STAGES; ++s) {
			mbar_init(bar_full + 8 * s, 5);                   // four warps that unpack, one that stages x
			mbar_init(bar_done + 8 * s, 1);                   // the unit's MMAs: sums are there, A and B are free
		}
		for (int s = 0; s < DC_W_RING; ++s) {
			mbar_init(bar_full_w + 8 * s, 2);                 // words; scales and zeros
			mbar_init(bar_empty_w + 8 * s, 4);
		}
		mbar_init(bar_fin, 1);
		*s_abort = 0;
		fence_mbar_init();
		tma_prefetch_desc(&tmw0);
		if (PAIR) tma_prefetch_desc(&tmw1);
	}
	if (warp == 2) {
		tmem_alloc(smem_u32(s_tmem), DC_TMEM_COLS);
		tmem_relinquish();
	}
	// rows that do not exist are zero for good
	for (int u = tid; u < DC_STAGES * DC_X_STAGE / 16; u += DC_THREADS) reinterpret_cast<uint4 *>(smem)[u] = make_uint4(0u, 0u, 0u, 0u);
	fence_proxy_async();
	tc_fence_before();
	__syncthreads();
	tc_fence_after();
	const uint32_t tmem_a = *s_tmem, tmem_d = tmem_a + DC_STAGES * 64;

	auto fail = [&](int code) {
		*s_abort = 1;
		atomicExch(p.status, code);
	};
	if (warp == 0 || warp == 3) {
		// ---------------- packed weights (warp 0), scales and zeros (warp 3); they depend on no earlier kernel ----------------
		// Two warps, and nothing but additions per unit: with one warp and a division the chain of these instructions was the bound
		// (8192 -> 16384, 16 rows: 25.0 us; without the division 22.0).
		const int nz = a.N >> 3, gk = a.groupsize >> 7;
		int s = 0, tile = (hi - 1) / np, left = n;
		uint32_t ph = 1, dst = sW, bar = bar_full_w;
		const uint32_t to_empty = bar_empty_w - bar_full_w;
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
				ok = dc_wait(bar + to_empty, ph, s_abort);
				if (!ok) break;
				if (one) {
					if (warp == 0) {
						mbar_arrive_expect_tx(bar, DC_W_SC);
						tma_load_2d(dst, &tmw0, n0, row, bar);
						if (PAIR) tma_load_2d(dst + 4096, &tmw1, n0, row, bar);
					} else {
						mbar_arrive_expect_tx(bar, DC_W_BYTES - DC_W_SC);
						dc_bulk_load(dst + DC_W_SC, sc0, TN * 2, bar);
						dc_bulk_load(dst + DC_W_QZ, qz0, TN / 2, bar);
						if (PAIR) {
							dc_bulk_load(dst + DC_W_SC + 128, sc1, TN * 2, bar);
							dc_bulk_load(dst + DC_W_QZ + 32, qz1, TN / 2, bar);
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
					dst = sW;
					bar = bar_full_w;
					ph ^= 1;
				}
			}
		}
		if (!ok) {
			fail(1);
			const unsigned long long t0 = global_timer_ns();          // copies in flight land before the CTA may end
			while (global_timer_ns() - t0 < 1000000ull) __nanosleep(1000);
		}
	} else if (warp == 1) {
		// ---------------- MMA issuer ----------------
		const uint32_t idesc = (1u << 4) | ((uint32_t)(16 >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);   // D fp32, A/B fp16 K-major, N = 16, M = 128
		uint64_t xd = smem_desc_sw128(sX);
		uint32_t ph = 0;
		int s = 0;
		const bool one = dc_elect();
		for (int i = 0; i < n; ++i) {
			if (!dc_wait(bar_full + 8 * s, ph, s_abort)) { fail(3); break; }
			tc_fence_after();
			if (one) {
				const uint32_t d = tmem_d + s * DC_D_COLS, at = tmem_a + s * 64;
				const uint64_t xs = xd + (uint64_t)(s * (DC_X_STAGE >> 4));
#pragma unroll
				for (int k = 0; k < 8; ++k) umma_f16_ts(d, at + 8 * k, xs + (uint64_t)((k >> 2) * 128 + 2 * (k & 3)), idesc, k ? 1u : 0u);
				umma_commit(bar_done + 8 * s);
			}
			__syncwarp();
			if (++s == DC_STAGES) {
				s = 0;
				ph ^= 1;
			}
		}
		if (one) umma_commit(bar_fin);
		__syncwarp();
	} else if (warp >= 4 && warp < 8) {
		// ---------------- x ----------------
		dec_stage_x<EPI, M8>(p, warp - 4, lane, sX, bar_full, bar_done, s_inv, s_abort);
	} else if (warp >= 8) {
		// ---------------- unpack, scale and add, epilogue ----------------
		const int q = warp & 3, grp = (warp - 8) >> 2, wt = q * 32 + lane, wid = tid - 256;      // tensor-memory lane = weight column of the tile
		const uint32_t w_off = PAIR ? (uint32_t)((wt >> 6) * 4096 + (wt & 63) * 4) : (uint32_t)(wt * 4);
		constexpr uint32_t W_ROW = PAIR ? 256 : 512;
		const uint32_t zsh = (wt & 7) * 4, quarter = (uint32_t)(q * 32) << 16;
		bool ok = true, waited = false;
		int i = grp, ws = grp;                              // next unit of this group, its stage of the packed ring
		uint32_t wp = 0;
		int tile = (hi - 1) / np, end = 0;                  // units of the segments so far
		while (end < n) {
			const int begin = end, k0 = max(lo - tile * np, 0), k1 = min(hi - tile * np, np);
			end += k1 - k0;
			float acc[ROWS];
#pragma unroll
			for (int r = 0; r < ROWS; ++r) acc[r] = 0.f;
			float sc1 = 0.f, sc2 = 0.f;                     // scales of the group's last unit and of the one before
			// sums of unit v (its stage, phase): tensor memory -> registers
			auto drain = [&](int v, float scale) {
				const int st = v % DC_STAGES;
				ok = ok && dc_wait(bar_done + 8 * st, (v / DC_STAGES) & 1, s_abort);
				if (!ok) return;
				tc_fence_after();
				float d[ROWS];
				if constexpr (M8) tmem_ld8(tmem_d + st * DC_D_COLS + quarter, d);
				else tmem_ld16(tmem_d + st * DC_D_COLS + quarter, d);
				tmem_ld_wait();
#pragma unroll
				for (int r = 0; r < ROWS; ++r) {
					asm volatile("" : "+f"(d[r]));              // not before the wait
					acc[r] = fmaf(scale, d[r], acc[r]);
				}
			};
			for (; i < end && ok; i += DC_GROUPS) {
				ok = dc_wait(bar_full_w + 8 * ws, wp, s_abort);
				if (!ok) break;
				if (i - DC_STAGES >= begin) drain(i - DC_STAGES, sc2);          // (an earlier segment's units have been drained)
				if (!ok) break;
				const uint32_t st = sW + ws * DC_W_STAGE, at = tmem_a + (i % DC_STAGES) * 64 + quarter;
				sc2 = sc1;
				sc1 = __half2float(__ushort_as_half((unsigned short)dc_lds16(st + DC_W_SC + wt * 2)));
				const uint32_t zz = ((dc_lds32(st + DC_W_QZ + (wt >> 3) * 4) >> zsh) & 0xFu) + 1u;
				const uint32_t ze = (0x6400u + zz) * 0x00010001u;            // half2(1024 + zero)
				const uint32_t zo = (0xD400u + (zz << 4)) * 0x00010001u;     // half2(-(64 + zero))
#pragma unroll
				for (int h = 0; h < 2; ++h) {
					uint32_t o[32];
#pragma unroll
					for (int r = 0; r < 8; ++r) {
						const uint32_t w = dc_lds32(st + w_off + (8 * h + r) * W_ROW), w8 = w >> 8;
						o[4 * r] = h2_sub(lop3_and_or(w, MASK_LO, MAGIC_1024), ze);                       // q - zero, exact: k0 k4
						o[4 * r + 1] = h2_fma(lop3_and_or(w, MASK_HI, MAGIC_1024), 0x2C002C00u, zo);      // k1 k5
						o[4 * r + 2] = h2_sub(lop3_and_or(w8, MASK_LO, MAGIC_1024), ze);                  // k2 k6
						o[4 * r + 3] = h2_fma(lop3_and_or(w8, MASK_HI, MAGIC_1024), 0x2C002C00u, zo);     // k3 k7
					}
					tmem_st32(at + 32 * h, o);
				}
				__syncwarp();
				if (lane == 0) mbar_arrive(bar_empty_w + 8 * ws);
				tmem_st_wait();
				tc_fence_before();
				__syncwarp();
				if (lane == 0) mbar_arrive(bar_full + 8 * (i % DC_STAGES));
				ws += DC_GROUPS;
				if (ws >= DC_W_RING) {
					ws -= DC_W_RING;
					wp ^= 1;
				}
			}
			if (i - 2 * DC_GROUPS >= begin) drain(i - 2 * DC_GROUPS, sc2);
			if (i - DC_GROUPS >= begin) drain(i - DC_GROUPS, sc1);
			tc_fence_before();
			if (!ok) fail(3);
#pragma unroll
			for (int r = 0; r < ROWS; ++r) red[(grp * ROWS + r) * 128 + wt] = acc[r];
			if (!waited) {
				pdl_wait();                                 // outputs, residual and the exchange area belong to earlier kernels until here
				waited = true;
			}
			dc_workers_sync();
			dec_finish<EPI, M8>(p, red, tile, k0, k1 < np, wid, s_abort);
			if (end < n) dc_workers_sync();                 // the tile in shared memory has been read
			--tile;
		}
	}
	tc_fence_before();
	__syncthreads();
	if (warp == 2) {
		// tensor memory goes back only after every MMA issued above has completed (also when unwinding)
		if (lane == 0) mbar_wait_bounded(bar_fin, 0, DC_SPIN);
		__syncwarp();
		tc_fence_after();
		tmem_dealloc(tmem_a, DC_TMEM_COLS);
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
	alignas(64) CUtensorMap tmw0, tmw1;
	if (int rc = dec_map(p.a.qw0, p.a.K, p.a.N, TN, &tmw0)) return rc;
	tmw1 = tmw0;
	if (EPI == DEC_EPI_SILU)
		if (int rc = dec_map(p.a.qw1, p.a.K, p.a.N, TN, &tmw1)) return rc;
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
	return cuda_status(cudaLaunchKernelEx(&cfg, k, tmw0, tmw1, p));
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
	const int grid = std::max(1, std::min({sms, DC_MAX_CTAS, p.units / 2}));          // at least two units each
	const bool m8 = a.M <= 8;
	switch (epi) {
		case DEC_EPI_PLAIN: return m8 ? dec_go<DEC_EPI_PLAIN, true>(p, grid, dev, stream) : dec_go<DEC_EPI_PLAIN, false>(p, grid, dev, stream);
		case DEC_EPI_SILU: return m8 ? dec_go<DEC_EPI_SILU, true>(p, grid, dev, stream) : dec_go<DEC_EPI_SILU, false>(p, grid, dev, stream);
		case DEC_EPI_ROPE: return m8 ? dec_go<DEC_EPI_ROPE, true>(p, grid, dev, stream) : dec_go<DEC_EPI_ROPE, false>(p, grid, dev, stream);
	}
	return GPTQ_ERR_INVALID;
}

}   // namespace gptq
