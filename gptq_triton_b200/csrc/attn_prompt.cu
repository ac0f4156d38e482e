// Attention of a prompt behind cached tokens with an additive mask [b, 1, t, S], head size 128, fp16: what QuantLlamaAttention.forward does between
// its two projections.
//
//   attn_prepare_kernel  classifies the 64 x 64 tiles of the mask (nothing visible / mixed / zero) and copies the cached rows in front of the new ones,
//                        which the projection writes in place: no concatenation
//   attn_prompt_kernel   one CTA of four warps per head and 64 queries; keys and values in tiles of 64, fetched asynchronously two deep; products on
//                        mma.m16n8k16, scores, softmax and sums in fp32.  Tiles in which nothing is visible are neither loaded nor computed, and
//                        the mask is read for mixed tiles only, so a causal mask costs half of the products and its diagonal.
//
// What bounds it: issue and latency of the legacy tensor path with eight warps per SM (220 TFLOP/s on long prompts), so a library kernel on the tcgen05 path is
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
constexpr float AP_LOG2E = 1.4426950408889634f;
enum { AP_HIDDEN = 0, AP_MIXED = 1, AP_OPEN = 2 };

struct PrepareParams {
	const __half *mask;
	long long mask_sb, mask_st;
	int mask_b, t, S, qt, kt;
	unsigned char *flags;                // [mask_b][qt][kt]
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
		bool hidden = true, open = true;
		if (row < p.t) {
			const unsigned short *src = reinterpret_cast<const unsigned short *>(p.mask) + mb * p.mask_sb + row * p.mask_st;
#pragma unroll
			for (int i = 0; i < 16; ++i) {
				if (col + i < p.S) {
					const unsigned short m = __ldg(src + col + i);
					hidden = hidden && m == 0xFC00u;                  // -infinity
					open = open && (m & 0x7FFFu) == 0;                // +- zero
				}
			}
		}
		hidden = __syncthreads_and(hidden);
		open = __syncthreads_and(open);
		if (threadIdx.x == 0) p.flags[id] = hidden ? AP_HIDDEN : open ? AP_OPEN : AP_MIXED;
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
	__half *out;                         // [b, t, heads * 128]
	int mask_b, heads, t, S, qt, kt;
	float scale;                         // times log2(e)
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

__global__ void __launch_bounds__(AP_THREADS, 2) attn_prompt_kernel(const PromptParams p) {
	extern __shared__ __align__(128) unsigned char ap_smem[];      // K, V of two tiles; queries
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, gid = lane >> 2, tig = lane & 3;
	const int pairs = gridDim.x / p.qt, late = blockIdx.x / pairs, pair = blockIdx.x - late * pairs;          // the longest of all heads first
	const int qt = p.qt - 1 - late, bi = pair / p.heads, head = pair - bi * p.heads;
	const int q0 = qt * AP_T, mb = p.mask_b == 1 ? 0 : bi;
	const uint32_t base = smem_u32(ap_smem), sq = base + 4 * AP_TILE;
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
	auto next = [&](int t) {
		while (t < p.kt && flags && flags[t] == AP_HIDDEN) ++t;
		return t;
	};
	load(sq, q, p.q_st, q0, p.t);
	int cur = next(0), buf = 0;
	if (cur < p.kt) {
		load(base, k, AP_D, cur * AP_T, p.S);
		load(base + AP_TILE, v, AP_D, cur * AP_T, p.S);
	}
	cp_async_commit();

	float o[16][4];
#pragma unroll
	for (int n = 0; n < 16; ++n) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f;
	float mx[2] = {-INFINITY, -INFINITY}, sum[2] = {0.f, 0.f};
	const int row = q0 + warp * 16 + gid;      // of o[.][0 .. 1]; row + 8 of o[.][2 .. 3]
#pragma unroll 1
	while (cur < p.kt) {
		const int kind = flags ? flags[cur] : (int)AP_MIXED, k0 = cur * AP_T, after = next(cur + 1);
		if (after < p.kt) {
			const uint32_t dst = base + (buf ^ 1) * 2 * AP_TILE;
			load(dst, k, AP_D, after * AP_T, p.S);
			load(dst + AP_TILE, v, AP_D, after * AP_T, p.S);
		}
		cp_async_commit();
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
		// scores in base 2 are s * f
		const float f = kind == AP_MIXED ? 1.f : p.scale;
		if (kind == AP_MIXED) {
			const __half *m0 = mask + (long long)min(row, p.t - 1) * p.mask_st, *m1 = mask + (long long)min(row + 8, p.t - 1) * p.mask_st;
#pragma unroll
			for (int n = 0; n < 8; ++n)
#pragma unroll
				for (int j = 0; j < 2; ++j) {
					const int key = min(k0 + n * 8 + 2 * tig + j, p.S - 1);
					s[n][j] = fmaf(s[n][j], p.scale, __half2float(m0[key]) * AP_LOG2E);
					s[n][2 + j] = fmaf(s[n][2 + j], p.scale, __half2float(m1[key]) * AP_LOG2E);
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
	p.scale = scale * AP_LOG2E;
	if ((long long)p.qt * heads * b > 0x7fffffff) return GPTQ_ERR_UNSUPPORTED;          // (more output than any memory holds)
	constexpr int smem = 5 * AP_TILE;
	if (cudaError_t e = cudaFuncSetAttribute(attn_prompt_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)) return cuda_status(e);
	return ap_launch(attn_prompt_kernel, dim3(p.qt * heads * b), AP_THREADS, smem, reinterpret_cast<cudaStream_t>(stream), p);
}

}   // extern "C"
