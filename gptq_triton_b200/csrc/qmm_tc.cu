// Prefill-regime (M > 16) quantised matmul on the 5th-generation tensor cores of sm_100a.
//
// The product is computed transposed, Y^T = deq(W)^T X^T: a weight column is a lane of tensor memory and the rows of X are the N
// of the MMA.  The dequantised weights are the A operand in TENSOR MEMORY, X is the B operand in shared memory.
//   - A thread that owns a column writes the 64 weights of a K-block with one tcgen05.st: no shared-memory stores, no proxy fence.
//     With both operands in shared memory the operand traffic was the bound of long prompts (176 KB per 256 x 256 x 64 block at
//     128 bytes per clock).
//   - The N of an MMA is any multiple of 16 up to 256, so a tile holds exactly the rows that there are: 40 rows cost 48, not 128.
// A CTA computes 128 columns (64 gate + 64 up columns for the fused MLP) x nr rows; K advances in blocks of 64.
//
//   warp 0      packed weights (8 words x 128 columns per K-block) by TMA into a deep ring; warp 3 their scales and zeros
//   warp 1      X tile [nr x 64] fp16, K-major, 128-byte swizzle
//   warp 2      MMA issuer: tcgen05.mma.cta_group::1.kind::f16, A from tensor memory, M = 128, N = nr, K = 16; one wait and one
//               commit per stage of one or two K-blocks
//   warp 3      also owns the tensor-memory allocation (nr columns of accumulators, 4 to 8 stages of 32 or 64 columns of weights)
//   warps 4-19  dequantise, four groups of four warps, group j serving the stages j, j + 4, ...: 8 packed words of a column
//               become 64 fp16 weights (q - zero) * scale with ONE rounding each, the weights of the dequantise-then-matmul path
// Afterwards the accumulators are turned through shared memory into an fp32 tile [row][128] and all warps run the epilogue:
// bias / residual, SiLU(gate) * up, or rotary + scatter to Q / K / V.
// Split K: the CTAs of a cluster take consecutive ranges of K-blocks of one tile; each then finishes its share of the rows,
// reading the partial tiles of the others from their shared memory in split order (deterministic; no pass through global memory).
//
// What bounds it: up to about 130 rows the issue slots of the dequantisation (17 instructions per 8 weights), above the MMAs and, from
// about 1000 rows, the power limit (1250 - 1430 TFLOP/s; cuBLAS bf16: 1670 in a burst, 1410 sustained).  Measured, in brackets the
// kernel with both operands in shared memory that this one replaced (us; 128-row tiles, split K through global memory):
//   M = 17    4096 -> 12288  13.8 (26.3)   22016 -> 8192  31.4 (56.2)   gate/up 8192 -> 2 x 22016   73 (190)
//   M = 203   4096 -> 12288  22.8 (46.8)   22016 -> 8192  60.6 (84.2)   gate/up 8192 -> 2 x 22016  130 (247)
//   M = 512   4096 -> 4096   17.9 (36.0)   11008 -> 4096  38.0 (55.8)   gate/up 4096 -> 2 x 11008   88 (132)
//   M = 2048  4096 -> 4096   55.8 (58.0)   11008 -> 4096   139 (145)    gate/up 4096 -> 2 x 11008  302 (332)
//
// It keeps its place in the stream in both directions: it stores many cache rows and may be the first reader of new weights, so it reads nothing
// ahead of its dependency wait and never triggers its successor (see pdl_trigger in common.cuh).  As a dependent launch it still has its
// barriers, tensor memory and launch latency behind it when the kernel in front ends: a layer of 512 rows 4096 -> 4096 takes 19.1 us per call,
// 20.5 as a plain launch; with weights ahead of the wait and an early trigger, which let attention read unfinished cache rows, it took 18.5.
//
// Every mbarrier wait is bounded; a wait that runs out sets a status word and the kernel unwinds (tensor memory is still released).
#include <algorithm>
#include <atomic>

#include <cuda.h>

#include "qmm_tc.cuh"
#include "tcgen05.cuh"

namespace gptq {

namespace {

constexpr int TC_BK = 64;
constexpr int TC_THREADS = 128 + 512;                       // producers, issuer, tensor-memory owner; 16 dequantise warps
constexpr int TC_MAX_NR = 256;                              // rows per tile (N of the MMA)
constexpr int TC_PAIR_NR = 144;                             // two K-blocks per stage up to this many rows (four stages fit)
constexpr int TC_TMEM_COLS = 512;
constexpr int TC_GROUPS = 4;                                // dequantise groups
// a packed stage of kp K-blocks: 8 kp words of 128 columns, scales and zeros of every K-block
__host__ __device__ constexpr int TC_W_SC(int kp) { return 4096 * kp; }
__host__ __device__ constexpr int TC_W_QZ(int kp) { return TC_W_SC(kp) + 256 * kp; }
__host__ __device__ constexpr int TC_W_STAGE(int kp) { return (TC_W_QZ(kp) + 64 * kp + 127) / 128 * 128; }
constexpr int TC_MAX_STAGES = 8, TC_MAX_WSTAGES = 20;
constexpr int TC_BARS = 2 * TC_MAX_STAGES + 2 * TC_MAX_WSTAGES + 1;
constexpr int TC_BAR_BYTES = (TC_BARS + 1) * 8;
constexpr int TC_SMEM = 227 * 1024;
constexpr uint32_t TC_SPIN = 1u << 24;
static_assert(4 * TC_MAX_NR * TC_BK * 2 + 16 * TC_W_STAGE(1) + TC_BAR_BYTES <= TC_SMEM, "shared memory per CTA, one K-block per stage");
static_assert(4 * TC_PAIR_NR * TC_BK * 2 * 2 + 8 * TC_W_STAGE(2) + TC_BAR_BYTES <= TC_SMEM, "shared memory per CTA, two");
static_assert(TC_MAX_NR + 4 * (TC_BK / 2) <= TC_TMEM_COLS && TC_PAIR_NR + 4 * TC_BK <= TC_TMEM_COLS, "tensor memory");

struct TcParams {
	TcArgs a;
	int *status;
	int nr;                      // rows per tile
	int kb_per_split;            // K-blocks per CTA
	int s_stages, w_stages;      // ring depths: X / dequantised weights (4 .. 8), packed weights (a multiple of 4)
	int bar_off;
	int out8;                    // rotary outputs may be stored 8 bytes at a time
};

// Wait of a whole warp: one poll inline, the bounded loop and the look at the abort flag out of line.  Every lane gets the same answer.
__device__ __noinline__ bool tc_wait_slow(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
	return __all_sync(0xffffffffu, !*abort_flag && mbar_wait_bounded(bar, parity, TC_SPIN));
}
__device__ __forceinline__ bool tc_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
	return __all_sync(0xffffffffu, mbar_try_wait(bar, parity)) || tc_wait_slow(bar, parity, abort_flag);
}
// the same without a call, for code with many live registers
__device__ __forceinline__ bool tc_wait_inline(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
	if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
	return __all_sync(0xffffffffu, !*abort_flag && mbar_wait_bounded(bar, parity, TC_SPIN));
}
__device__ __forceinline__ bool tc_elect() {
	uint32_t r;
	asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xFFFFFFFF;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
	return r != 0;
}
__device__ __forceinline__ void tc_bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
	asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ uint32_t tc_lds32(uint32_t addr) {
	uint32_t r;
	asm volatile("ld.shared.u32 %0, [%1];" : "=r"(r) : "r"(addr) : "memory");
	return r;
}
__device__ __forceinline__ uint32_t tc_lds16(uint32_t addr) {
	unsigned short r;
	asm volatile("ld.shared.u16 %0, [%1];" : "=h"(r) : "r"(addr) : "memory");
	return r;
}
__device__ __forceinline__ float4 tc_lds128(uint32_t addr) {
	float4 r;
	asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w) : "r"(addr) : "memory");
	return r;
}
// four floats at this CTA's address `addr`, in the shared memory of CTA `rank` of the cluster
__device__ __forceinline__ float4 tc_ld_peer(uint32_t addr, uint32_t rank) {
	float4 r;
	asm volatile(
		"{\n\t.reg .b32 a;\n\t"
		"mapa.shared::cluster.u32 a, %4, %5;\n\t"
		"ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [a];\n\t}"
		: "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w)
		: "r"(addr), "r"(rank)
		: "memory");
	return r;
}
__device__ __forceinline__ void tc_cluster_sync() {
	asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

}   // namespace

}   // namespace gptq

#include "qmm_tc_kernel.inl"

// ---- host side -------------------------------------------------------------------------------
namespace gptq {

EncodeTiledFn tensor_map_encoder();      // defined in api.cu
bool pdl_enabled();
int g_tc_force = 0;                    // tests: 0 = choose by cost, 1 .. 4 = at most 64, 128, 192, 256 rows per tile
extern "C" void gptq_debug_tc_force(int cfg) { g_tc_force = cfg; }

bool tc_shape_ok(int M, int K, int N, int groupsize) {
	return M > 16 && N % 128 == 0 && K % TC_BK == 0 && groupsize % TC_BK == 0 && K % groupsize == 0;
}

size_t tc_ws_bytes(int, int) { return 16384; }      // the status word at the end of the first 16 KB
int g_tc_splitk = 0;                   // tests: 0 = choose by cost, n = force n splits
extern "C" void gptq_debug_tc_splitk(int n) { g_tc_splitk = n; }

static int tc_map(const void *base, CUtensorMapDataType type, int elem, cuuint64_t cols, cuuint64_t rows, cuuint64_t ld, cuuint32_t box_cols, cuuint32_t box_rows,
				  CUtensorMapSwizzle swizzle, CUtensorMap *out) {
	EncodeTiledFn enc = tensor_map_encoder();
	if (!enc) return GPTQ_ERR_CUDA;
	cuuint64_t dims[2] = {cols, rows}, strides[1] = {ld * elem};
	cuuint32_t box[2] = {box_cols, box_rows}, estr[2] = {1, 1};
	CUresult r = enc(out, type, 2, const_cast<void *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
					 CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
	if (r != CUDA_SUCCESS) {
		g_last_cuda_error = (int)r;
		return GPTQ_ERR_CUDA;
	}
	return GPTQ_OK;
}

constexpr int TC_MAX_SPLITS = 8;       // portable cluster size
// Estimated time of a CTA in us, fitted to measurements (M = 17 .. 2048, K = 4096 / 8192 / 11008 / 22016): a K-block costs the
// dequantisation (0.16 us at 32 rows in stages of two, 0.22 in stages of one) or the MMAs (0.38 us at 256 rows), a tile 2.5 us to start and
// drain; with split K the partial tiles of the cluster are summed through distributed shared memory (4 us at 32 rows, 7 us at 256).  Against 4.8 us at 32
// rows, a first fit on K >= 4096 only, us (dependent launches): 1024 -> 1024, 40 rows 5.9 -> 5.4; 2048 -> 6144, 17 rows 9.2 -> 8.4; 2048 -> 3072, 203 rows 10.1 -> 9.5;
// 3072 -> 3072, 203 rows 11.4 -> 10.6; 2560 -> 7680, 100 rows 11.6 -> 10.7; 5504 -> 2048, 512 rows 16.6 -> 15.2; the wide layers choose as before.  That holds for
// one wave of clusters; of more the first fit is the better one (whole clusters have to leave before the next start): 8192 -> 10240, 64 rows 25.2 without a split, 26.8
// with one, 8192 -> 2 x 5504, 100 rows 28.1 / 30.2.
static double tc_cta_us(int nr, int splits, int kblocks, bool one_wave) {
	const double t_kb = nr <= TC_PAIR_NR ? 0.14 + 0.00065 * nr : std::max(0.22 + 0.0002 * nr, 0.0015 * nr);
	return kblocks * t_kb + (splits == 1 ? 2.5 : one_wave ? 3.5 + 0.014 * nr : 4.5 + 0.01 * nr);
}

template <int EPI, int KP>
static int tc_ready(int dev) {
	static std::atomic<bool> ready[64];
	if (!ready[dev]) {
		cudaError_t e = cudaFuncSetAttribute(tc_kernel<EPI, KP>, cudaFuncAttributeMaxDynamicSharedMemorySize, TC_SMEM);
		if (e != cudaSuccess) return cuda_status(e);
		ready[dev] = true;
	}
	return GPTQ_OK;
}

static void tc_attrs(cudaLaunchConfig_t &cfg, cudaLaunchAttribute *attr, int splits, bool pdl) {
	cfg.blockDim = dim3(TC_THREADS);
	cfg.attrs = attr;
	cfg.numAttrs = 0;
	if (splits > 1) {
		cudaLaunchAttribute &c = attr[cfg.numAttrs++];
		c.id = cudaLaunchAttributeClusterDimension;
		c.val.clusterDim.x = 1;
		c.val.clusterDim.y = 1;
		c.val.clusterDim.z = splits;
	}
	if (pdl) {
		cudaLaunchAttribute &c = attr[cfg.numAttrs++];
		c.id = cudaLaunchAttributeProgrammaticStreamSerialization;
		c.val.programmaticStreamSerializationAllowed = 1;
	}
}

template <int EPI, int KP>
static int tc_go(TcParams p, int splits, int dev, cudaStream_t stream) {
	constexpr int TN = EPI == TC_EPI_SILU ? 64 : 128;
	const TcArgs &a = p.a;
	if (int rc = tc_ready<EPI, KP>(dev)) return rc;
	// rings: X and the dequantised weights share their stages, bounded by shared and by tensor memory
	const int x_stage = p.nr * TC_BK * 2 * KP, left = TC_SMEM - TC_BAR_BYTES, w_min = KP == 2 ? 8 : 16;
	p.s_stages = std::min({TC_MAX_STAGES, (left - w_min * TC_W_STAGE(KP)) / x_stage, (TC_TMEM_COLS - p.nr) / (KP * TC_BK / 2)});
	p.w_stages = std::min(TC_MAX_WSTAGES, (left - p.s_stages * x_stage) / TC_W_STAGE(KP)) & ~3;
	p.bar_off = p.s_stages * x_stage + p.w_stages * TC_W_STAGE(KP);
	alignas(64) CUtensorMap tmx, tmw0, tmw1;
	if (int rc = tc_map(a.x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, a.K, a.M, a.ldx, TC_BK, p.nr, CU_TENSOR_MAP_SWIZZLE_128B, &tmx)) return rc;
	if (int rc = tc_map(a.qw0, CU_TENSOR_MAP_DATA_TYPE_INT32, 4, a.N, a.K / 8, a.N, TN, 8 * KP, CU_TENSOR_MAP_SWIZZLE_NONE, &tmw0)) return rc;
	tmw1 = tmw0;
	if (EPI == TC_EPI_SILU)
		if (int rc = tc_map(a.qw1, CU_TENSOR_MAP_DATA_TYPE_INT32, 4, a.N, a.K / 8, a.N, TN, 8 * KP, CU_TENSOR_MAP_SWIZZLE_NONE, &tmw1)) return rc;
	cudaLaunchConfig_t cfg = {};
	cudaLaunchAttribute attr[2];
	tc_attrs(cfg, attr, splits, pdl_enabled());
	cfg.stream = stream;
	cfg.gridDim = dim3((a.M + p.nr - 1) / p.nr, a.N / TN, splits);
	cfg.dynamicSmemBytes = p.bar_off + TC_BAR_BYTES;
	return cuda_status(cudaLaunchKernelEx(&cfg, tc_kernel<EPI, KP>, tmx, tmw0, tmw1, p));
}

template <int EPI>
static int tc_launch_inst(TcParams p, cudaStream_t stream) {
	constexpr int TN = EPI == TC_EPI_SILU ? 64 : 128;
	const TcArgs &a = p.a;
	int dev = 0;
	if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return GPTQ_ERR_CUDA;
	if (int rc = tc_ready<EPI, 1>(dev)) return rc;
	// CTAs that run at the same time: one per SM, in whole clusters
	static std::atomic<int> slots[64][TC_MAX_SPLITS + 1];
	auto slots_of = [&](int splits) -> int {
		int n = slots[dev][splits];
		if (n) return n;
		if (splits == 1) {
			if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) n = 148;
		} else {
			cudaLaunchConfig_t cfg = {};
			cudaLaunchAttribute attr[2];
			tc_attrs(cfg, attr, splits, false);
			cfg.gridDim = dim3(1, 1, splits);
			cfg.dynamicSmemBytes = TC_SMEM;
			int clusters = 0;
			if (cudaOccupancyMaxActiveClusters(&clusters, tc_kernel<EPI, 1>, &cfg) != cudaSuccess) {
				cudaGetLastError();
				clusters = 0;
			}
			n = clusters > 0 ? clusters * splits : -1;          // -1: such clusters do not fit
		}
		slots[dev][splits] = n;
		return n;
	};
	// Rows per tile and splits by estimated time: waves of CTAs times the time of one.
	const int nkb = a.K / TC_BK, tiles = a.N / TN;
	const int cap = g_tc_force ? std::min(TC_MAX_NR, 64 * g_tc_force) : TC_MAX_NR;
	const int mt_min = (a.M + cap - 1) / cap;
	double best = 1e30;
	int best_splits = 1;
	for (int mt = mt_min; mt <= mt_min + (g_tc_force ? 0 : 3); ++mt) {
		const int nr = ((a.M + mt - 1) / mt + 15) & ~15;
		if ((mt - 1) * nr >= a.M) break;                                 // an empty tile
		for (int splits = 1; splits <= std::min(TC_MAX_SPLITS, nkb); ++splits) {
			const int per = splits == 1 ? nkb : ((nkb + splits - 1) / splits + 1) & ~1;      // whole stages
			if ((splits - 1) * per >= nkb) continue;                     // an empty split
			if (g_tc_splitk > 0 ? splits != g_tc_splitk : splits > 1 && per < 4) continue;
			const int n = slots_of(splits);
			if (n <= 0) continue;
			const long long ctas = (long long)mt * tiles * splits;
			// (two tiles of 16 rows unpack the same weights twice for next to no MMAs: not for a tie; 2560 -> 2048, 17 rows 5.9 / 6.4)
			const double t = (double)((ctas + n - 1) / n) * tc_cta_us(nr, splits, per, ctas <= n) * (mt > 1 && nr <= 16 ? 1.02 : 1.0);
			if (t < best) {
				best = t;
				best_splits = splits;
				p.nr = nr;
				p.kb_per_split = per;
			}
		}
	}
	if (best >= 1e30) {          // a forced split that is not possible: none
		p.nr = ((a.M + mt_min - 1) / mt_min + 15) & ~15;
		p.kb_per_split = nkb;
	}
	return p.nr <= TC_PAIR_NR ? tc_go<EPI, 2>(p, best_splits, dev, stream) : tc_go<EPI, 1>(p, best_splits, dev, stream);
}

int tc_launch(const TcArgs &a, int epi, void *workspace, size_t ws_bytes, cudaStream_t stream) {
	if (a.perm) return GPTQ_ERR_UNSUPPORTED;
	if (!workspace || ws_bytes < 16384) return GPTQ_ERR_WORKSPACE;
	if (a.ldx % 8 != 0) return GPTQ_ERR_ALIGN;
	TcParams p = {};
	p.a = a;
	p.status = reinterpret_cast<int *>(workspace) + (16384 / 4 - 1);
	if (epi == TC_EPI_ROPE) {
		auto even = [](const void *ptr) { return (reinterpret_cast<uintptr_t>(ptr) & 7u) == 0; };
		p.out8 = even(a.q_out) && even(a.k_out) && even(a.v_out) && ((a.q_stride_m | a.kv_sb | a.kv_st | a.kv_sh | a.kv_sp) & 3) == 0;
	}
	switch (epi) {
		case TC_EPI_PLAIN: return tc_launch_inst<TC_EPI_PLAIN>(p, stream);
		case TC_EPI_SILU: return tc_launch_inst<TC_EPI_SILU>(p, stream);
		case TC_EPI_ROPE: return tc_launch_inst<TC_EPI_ROPE>(p, stream);
	}
	return GPTQ_ERR_INVALID;
}

}   // namespace gptq
