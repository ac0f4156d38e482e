// Decode-regime projection (M <= 8 rows) over dense weights [N, K], HBM-bound: every weight is read once with 16-byte loads
// straight into registers, double-buffered so that loads are always in flight across tile boundaries.
//
// A CTA of 8 warps owns tiles of 16 weight rows (strided over the grid) and splits K over its warps.  bf16: the weight rows
// are the A operand of mma.m16n8k16 and the activations the B operand.  A dot product does not care about the order of k, so
// lane (gid, tig) feeds the eight consecutive k that its 16-byte loads deliver for rows gid and gid + 8 and the same eight k
// of activation row gid: two MMAs per pair of loads, no shuffle.  fp32: the same layout on the FMA units.
// bf16 and few rows: dense_ring_kernel below, the same with the weights in shared memory.
// Few tiles (a narrow projection) leave most SMs idle: then a cluster of CTAs shares a tile's K, the partial sums meet in the first
// CTA's shared memory.
// The prologue optionally prepares the rows itself (embedding lookup, residual, norm), the epilogue applies what
// follows the projection (rotary queries / raw latent / gates, act(gate) * up, scaled logits with the greedy choice).
#include <algorithm>

#include <cuda.h>

#include "dense.cuh"

namespace gptq {

int dense_tensor_map(const void *base, long long rows, long long cols, long long ld, int box_rows, int box_cols, CUtensorMap *out);      // dense_tc.cu

namespace {

constexpr int SK_M = 8, SK_U = 4, SK_REDLD = 17, SK_PARTS = 8;
constexpr size_t SK_STATIC = (2 * DN_WARPS * SK_M * SK_REDLD + RP_SMEM) * sizeof(float) + 64;
constexpr size_t SK_SMEM_MAX = 227 * 1024 - SK_STATIC - 1024;

// Results va, vb of pair j of activation row m in a tile of 16 weight rows.
template <typename T>
__device__ __forceinline__ void finish_pair(const DenseArgs &p, int m, int j, int tile, float va, float vb, unsigned long long &best) {
	if (p.e.mode == DENSE_EPI_GATED) {
		Elem<T>::store(reinterpret_cast<T *>(p.e.out) + (size_t)m * p.e.ldo + tile * 8 + j, activation(p.e.act, va) * vb);
		return;
	}
	const int n = tile * 16 + 2 * j;
	epi_pair<T>(p.e, m, n, va, vb);
	if (p.e.mode == DENSE_EPI_LOGITS) {
		if (n < p.N) best = max(best, argmax_key(va * p.e.scale, n));
		if (n + 1 < p.N) best = max(best, argmax_key(vb * p.e.scale, n + 1));
	}
}

// Greedy choice: one candidate per CTA and row (best: running candidate of thread (m = tid / 8)), the last CTA writes token and position.
__device__ __forceinline__ void choose(const DenseArgs &p, unsigned long long best, int *s_last) {
	if (p.e.mode != DENSE_EPI_LOGITS || !p.e.best) return;
	const int tid = threadIdx.x;
	if (tid < 8 * SK_M) {                        // whole warps
#pragma unroll
		for (int s = 1; s < 8; s <<= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, s));
		if (tid < 8 * p.M && (tid & 7) == 0) atomicMax(p.e.best + (tid >> 3), best);
	}
	__syncthreads();
	if (tid == 0) {
		unsigned t;
		asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(t) : "l"(p.e.ticket) : "memory");
		*s_last = t == gridDim.x - 1;
		if (*s_last) *p.e.ticket = 0u;
	}
	__syncthreads();
	if (*s_last && tid < p.M) {
		const unsigned long long b = atomicExch(p.e.best + tid, 0ull);
		p.e.tok[tid] = (int64_t)(uint32_t)~(uint32_t)b;
		p.e.pos_inout[tid] += 1;
	}
}

template <typename T, bool SPLIT>
__global__ void __launch_bounds__(DN_THREADS, 2) dense_skinny_kernel(const DenseArgs p, int kparts) {
	constexpr int E = 16 / sizeof(T);            // elements per 16-byte load
	constexpr int STEP = 4 * E;                  // k per step of a warp
	extern __shared__ __align__(16) unsigned char sk_smem[];
	__shared__ float s_red[2][DN_WARPS][SK_M][SK_REDLD];
	__shared__ float s_norm[RP_SMEM];
	__shared__ int s_last;
	__shared__ float2 s_part[SPLIT ? SK_PARTS : 1][SPLIT ? 8 * SK_M : 1];
	if (SPLIT) cluster_arrive();                 // (every CTA of the cluster runs before its shared memory is written)
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, gid = lane >> 2, tig = lane & 3;
	const int xs = p.K * (int)sizeof(T) + 16;    // bytes per staged row
	const int rank = SPLIT ? (int)cluster_rank() : 0, tile0 = SPLIT ? (int)blockIdx.x / kparts : (int)blockIdx.x, stride = SPLIT ? (int)gridDim.x / kparts : (int)gridDim.x;
	const int slots = DN_WARPS * (SPLIT ? kparts : 1);
	const int nsteps = (p.K + STEP - 1) / STEP, spw = (nsteps + slots - 1) / slots;
	const int s0 = min((rank * DN_WARPS + warp) * spw, nsteps), s1 = min(s0 + spw, nsteps);
	const int nbatch = (spw + SK_U - 1) / SK_U;
	const int ntiles = (p.N + 15) >> 4;
	const int mytiles = (ntiles - tile0 + stride - 1) / stride;          // (SPLIT: one)
	const int total = mytiles * nbatch;
	const T *w = reinterpret_cast<const T *>(p.w);

	uint4 wa[2][SK_U], wb[2][SK_U];
	auto load = [&](int it, uint4 (&a)[SK_U], uint4 (&b)[SK_U]) {
		const int ti = it / nbatch, bi = it - ti * nbatch;
		const int row = (tile0 + ti * stride) * 16 + gid;
		const T *pa = w + (size_t)min(row, p.N - 1) * p.ldw, *pb = w + (size_t)min(row + 8, p.N - 1) * p.ldw;
#pragma unroll
		for (int u = 0; u < SK_U; ++u) {
			const int s = s0 + bi * SK_U + u, k = s * STEP + tig * E;
			if (s < s1 && k < p.K) {
				a[u] = ld_nc_v4(pa + k);
				b[u] = ld_nc_v4(pb + k);
			} else {
				a[u] = make_uint4(0u, 0u, 0u, 0u);
				b[u] = a[u];
			}
		}
	};
	load(0, wa[0], wb[0]);                       // weights do not depend on earlier kernels
	pdl_wait();
	pdl_trigger();

	// ---- stage the rows -------------------------------------------------------------------------------------------
	if (p.prep) {
		for (int m = 0; m < p.M; ++m) {
			if (m) __syncthreads();
			prepare_row<T>(p.rp, m, reinterpret_cast<T *>(sk_smem + (size_t)m * xs), p.rp.x_out != nullptr && blockIdx.x == 0, s_norm);
		}
	} else {
		const int units = p.K / E;
		for (int m = 0; m < p.M; ++m) {
			const uint4 *src = reinterpret_cast<const uint4 *>(reinterpret_cast<const T *>(p.x) + (size_t)m * p.ldx);
			for (int u = tid; u < units; u += DN_THREADS) *reinterpret_cast<uint4 *>(sk_smem + (size_t)m * xs + u * 16) = __ldcg(src + u);
		}
	}
	__syncthreads();

	float d[4] = {0.f, 0.f, 0.f, 0.f};           // bf16 accumulators
	float f[2][SK_M];                            // fp32 accumulators: rows gid, gid + 8 by activation row
#pragma unroll
	for (int m = 0; m < SK_M; ++m) f[0][m] = f[1][m] = 0.f;
	const unsigned char *xrow = sk_smem + (size_t)min(gid, p.M - 1) * xs;
	const bool live = gid < p.M;
	unsigned long long best = 0ull;              // LOGITS: running candidate of thread (m = tid / 8)

	float part_a = 0.f, part_b = 0.f;            // SPLIT: this CTA's share of the results of threads below 8 M
	auto finish = [&](int m, int j, int tile, float va, float vb) { finish_pair<T>(p, m, j, tile, va, vb, best); };
	auto compute = [&](int it, uint4 (&a)[SK_U], uint4 (&b)[SK_U]) {
		const int ti = it / nbatch, bi = it - ti * nbatch;
#pragma unroll
		for (int u = 0; u < SK_U; ++u) {
			const int s = s0 + bi * SK_U + u, k = min(s * STEP + tig * E, p.K - E);      // beyond the range the weights are zero
			if (sizeof(T) == 2) {
				uint4 x = make_uint4(0u, 0u, 0u, 0u);
				if (live) x = *reinterpret_cast<const uint4 *>(xrow + k * 2);
				mma16816_bf16(d, a[u].x, b[u].x, a[u].y, b[u].y, x.x, x.y);
				mma16816_bf16(d, a[u].z, b[u].z, a[u].w, b[u].w, x.z, x.w);
			} else {
#pragma unroll
				for (int m = 0; m < SK_M; ++m) {
					if (m < p.M) {
						const float4 x = *reinterpret_cast<const float4 *>(sk_smem + (size_t)m * xs + k * 4);
						f[0][m] = fmaf(__uint_as_float(a[u].x), x.x, fmaf(__uint_as_float(a[u].y), x.y, fmaf(__uint_as_float(a[u].z), x.z, fmaf(__uint_as_float(a[u].w), x.w, f[0][m]))));
						f[1][m] = fmaf(__uint_as_float(b[u].x), x.x, fmaf(__uint_as_float(b[u].y), x.y, fmaf(__uint_as_float(b[u].z), x.z, fmaf(__uint_as_float(b[u].w), x.w, f[1][m]))));
					}
				}
			}
		}
		if (bi != nbatch - 1) return;
		// ---- end of a tile: sum the warps' K slices (fixed order), epilogue ----------------------------------------
		float(*red)[SK_M][SK_REDLD] = s_red[ti & 1];
		if (sizeof(T) == 2) {
			const int c = 2 * tig;
			if (c < p.M) {
				red[warp][c][gid] = d[0];
				red[warp][c][gid + 8] = d[2];
			}
			if (c + 1 < p.M) {
				red[warp][c + 1][gid] = d[1];
				red[warp][c + 1][gid + 8] = d[3];
			}
			d[0] = d[1] = d[2] = d[3] = 0.f;
		} else {
#pragma unroll
			for (int m = 0; m < SK_M; ++m) {
				if (m < p.M) {
#pragma unroll
					for (int r = 0; r < 2; ++r) {
						float v = f[r][m];
						v += __shfl_xor_sync(0xffffffffu, v, 1);
						v += __shfl_xor_sync(0xffffffffu, v, 2);
						if (tig == 0) red[warp][m][gid + 8 * r] = v;
						f[r][m] = 0.f;
					}
				}
			}
		}
		__syncthreads();                         // the buffer is written again two tiles later, behind the next tile's barrier
		if (tid < 8 * p.M) {
			const int m = tid >> 3, j = tid & 7, tile = tile0 + ti * stride;
			const bool gated = p.e.mode == DENSE_EPI_GATED;
			const int ra = gated ? j : 2 * j, rb = gated ? j + 8 : 2 * j + 1;
			float va = 0.f, vb = 0.f;
#pragma unroll
			for (int i = 0; i < DN_WARPS; ++i) {
				va += red[i][m][ra];
				vb += red[i][m][rb];
			}
			if (SPLIT) {
				part_a = va;
				part_b = vb;
			} else {
				finish(m, j, tile, va, vb);
			}
		}
	};
#pragma unroll 1
	for (int it = 0; it < total; it += 2) {
		if (it + 1 < total) load(it + 1, wa[1], wb[1]);
		compute(it, wa[0], wb[0]);
		if (it + 2 < total) load(it + 2, wa[0], wb[0]);
		if (it + 1 < total) compute(it + 1, wa[1], wb[1]);
	}

	if (SPLIT) {
		__syncwarp();
		cluster_wait();
		if (tid < 8 * p.M) cluster_store2(cluster_map(smem_u32(&s_part[rank][tid]), 0), part_a, part_b);
		__syncwarp();
		cluster_arrive();
		cluster_wait();
		if (rank == 0 && tid < 8 * p.M) {
			float va = 0.f, vb = 0.f;
			for (int i = 0; i < kparts; ++i) {
				va += s_part[i][tid].x;
				vb += s_part[i][tid].y;
			}
			finish(tid >> 3, tid & 7, tile0, va, vb);
		}
		return;
	}
	choose(p, best, &s_last);
}

// The same for up to RG_ROWS rows in bf16, with the weights on their way in shared memory instead of registers: every warp streams its K slice of the
// tiles through a ring of its own (boxes of 16 rows x 64 k by TMA, 128-byte swizzle).  Five boxes of 2 KB for each of eight warps keep 80 KB in flight
// per SM, twice what the registers hold, and the ring is full before the launch in front ends.
// Bound: HBM for wide layers (32000 x 2048: 24.3 us = 5.4 TB/s alone), else the chain wait - rows - sums - store of about 4.5 us per launch.  In a step
// (2048 hidden): down 9.2 -> 5.4 us, gate/up 13.0 -> 11.1, out 4.9 -> 4.6; the step 433 -> 400 us, of the state-space model 273 -> 251, and with the norm weights ahead
// of the wait (RowWeights) 381 and 240.
// One CTA per SM, by the shared memory that it asks for: with two resident CTAs per SM, so that the next launch's rings could fill beside this
// one, the scheduler puts two CTAs of one launch on some SMs and none on others (head 31 -> 67 us, step 482).  More stages are slower (10: 417),
// and SMs left free for the next launch change nothing (148 / 144 / 140 CTAs: 382 / 384 / 384; 3 layers of 4096 313 / 314 / 324).
constexpr int RG_ROWS = 5, RG_STAGES = 5, RG_BOX = 2048, RG_MIN_SMEM = 120 * 1024;
constexpr int RG_STATIC = (2 * DN_WARPS * SK_M * SK_REDLD + RP_SMEM) * (int)sizeof(float) + DN_WARPS * RG_STAGES * 8 + 64 + 1024;

// One verdict for the whole warp, which goes on to MMAs and shares the stage.  (192 registers: the next launch's CTA of 256 threads with 64 each fits beside this kernel's;
// with 194, the slow path out of line, a request of the state-space model took 7.15 instead of 7.05 ms.)
__device__ __forceinline__ bool rg_wait(uint32_t bar, uint32_t parity) { return __all_sync(0xffffffffu, mbar_wait_bounded(bar, parity)); }

__global__ void __launch_bounds__(DN_THREADS, 1) dense_ring_kernel(const __grid_constant__ CUtensorMap tmw, const __grid_constant__ DenseArgs p, int stages) {
	extern __shared__ __align__(1024) unsigned char rg_smem[];
	__shared__ float s_red[2][DN_WARPS][SK_M][SK_REDLD];
	__shared__ float s_norm[RP_SMEM];
	__shared__ __align__(8) uint64_t s_bar[DN_WARPS][RG_STAGES];
	__shared__ int s_last;
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, gid = lane >> 2, tig = lane & 3;
	const int nunits = (p.K + 63) >> 6, upw = (nunits + DN_WARPS - 1) / DN_WARPS, u0 = min(warp * upw, nunits), count = min(u0 + upw, nunits) - u0;
	const int xs = nunits * 128 + 16;            // bytes per staged row
	const int ntiles = (p.N + 15) >> 4, mytiles = (ntiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
	unsigned char *rows = rg_smem + (size_t)DN_WARPS * stages * RG_BOX;
	const uint32_t ring = smem_u32(rg_smem) + warp * stages * RG_BOX, bars = smem_u32(s_bar[warp]);

	if (lane == 0) {
		for (int s = 0; s < stages; ++s) mbar_init(bars + 8 * s, 1);
		fence_mbar_init();
		tma_prefetch_desc(&tmw);
	}
	__syncwarp();
	int left = mytiles * count, pu = 0, prow = blockIdx.x * 16, ps = 0;          // boxes to load, unit and row of the next one, its stage
	auto load = [&]() {
		if (left == 0) return;
		--left;
		if (lane == 0) {
			mbar_arrive_expect_tx(bars + 8 * ps, RG_BOX);
			tma_load_2d(ring + ps * RG_BOX, &tmw, (u0 + pu) * 64, prow, bars + 8 * ps);
		}
		if (++ps == stages) ps = 0;
		if (++pu == count) {
			pu = 0;
			prow += gridDim.x * 16;
		}
	};
#pragma unroll 1
	for (int s = 0; s < stages; ++s) load();     // weights do not depend on earlier kernels
	RowWeights weights;
	if (p.prep) weights.load(p.rp);
	pdl_wait();
	pdl_trigger();

	// ---- stage the rows, zeros up to a multiple of 64 ----------------------------------------------------------------
	if (p.prep) {
		for (int m = 0; m < p.M; ++m) {
			if (m) __syncthreads();
			prepare_row<bf16, true>(p.rp, m, reinterpret_cast<bf16 *>(rows + (size_t)m * xs), p.rp.x_out != nullptr && blockIdx.x == 0, s_norm, &weights);
		}
	} else {
		const int units = p.K / 8;
		for (int m = 0; m < p.M; ++m)            // asynchronous copies (through L2): all rows in flight at once
			for (int u = tid; u < units; u += DN_THREADS) cp_async16(rows + (size_t)m * xs + u * 16, reinterpret_cast<const bf16 *>(p.x) + (size_t)m * p.ldx + u * 8);
		cp_async_commit();
		cp_async_wait<0>();
	}
	const int pad = nunits * 8 - p.K / 8;        // 16-byte units behind the last k
	if (tid < pad * p.M) *reinterpret_cast<uint4 *>(rows + (size_t)(tid / pad) * xs + (p.K / 8 + tid % pad) * 16) = make_uint4(0u, 0u, 0u, 0u);
	__syncthreads();

	const bool live = gid < p.M;
	const unsigned char *xrow = rows + (size_t)(live ? gid : 0) * xs + u0 * 128 + tig * 16;
	const uint32_t a0 = ring + gid * 128 + ((tig ^ gid) << 4), a1 = ring + gid * 128 + (((4 + tig) ^ gid) << 4);
	unsigned long long best = 0ull;
	bool ok = true;
	int cs = 0;
	uint32_t parity = 0;
#pragma unroll 1
	for (int ti = 0; ti < mytiles; ++ti) {
		float d[4] = {0.f, 0.f, 0.f, 0.f}, e[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
		for (int u = 0; u < count; ++u) {
			if (ok && !rg_wait(bars + 8 * cs, parity)) {
				ok = false;
				left = 0;                                // no further copies; the sums are worthless, the status says so
			}
			uint4 x0 = make_uint4(0u, 0u, 0u, 0u), x1 = x0;
			if (live) {
				x0 = *reinterpret_cast<const uint4 *>(xrow + u * 128);
				x1 = *reinterpret_cast<const uint4 *>(xrow + u * 128 + 64);
			}
			uint4 w[4];
#pragma unroll
			for (int i = 0; i < 4; ++i)
				asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(w[i].x), "=r"(w[i].y), "=r"(w[i].z), "=r"(w[i].w) : "r"((i & 2 ? a1 : a0) + cs * RG_BOX + (i & 1) * 1024) : "memory");
			mma16816_bf16(d, w[0].x, w[1].x, w[0].y, w[1].y, x0.x, x0.y);
			mma16816_bf16(e, w[2].x, w[3].x, w[2].y, w[3].y, x1.x, x1.y);
			mma16816_bf16(d, w[0].z, w[1].z, w[0].w, w[1].w, x0.z, x0.w);
			mma16816_bf16(e, w[2].z, w[3].z, w[2].w, w[3].w, x1.z, x1.w);
			__syncwarp();
			load();                                  // the stage just read is the oldest
			if (++cs == stages) {
				cs = 0;
				parity ^= 1u;
			}
		}
		float(*red)[SK_M][SK_REDLD] = s_red[ti & 1];
		const int c = 2 * tig;
		if (c < p.M) {
			red[warp][c][gid] = d[0] + e[0];
			red[warp][c][gid + 8] = d[2] + e[2];
		}
		if (c + 1 < p.M) {
			red[warp][c + 1][gid] = d[1] + e[1];
			red[warp][c + 1][gid + 8] = d[3] + e[3];
		}
		__syncthreads();                         // the buffer is written again two tiles later, behind the next tile's barrier
		if (tid < 8 * p.M) {
			const int m = tid >> 3, j = tid & 7;
			const bool gated = p.e.mode == DENSE_EPI_GATED;
			const int ra = gated ? j : 2 * j, rb = gated ? j + 8 : 2 * j + 1;
			float va = 0.f, vb = 0.f;
#pragma unroll
			for (int i = 0; i < DN_WARPS; ++i) {
				va += red[i][m][ra];
				vb += red[i][m][rb];
			}
			finish_pair<bf16>(p, m, j, blockIdx.x + ti * gridDim.x, va, vb, best);
		}
	}
	if (!ok) {
		if (lane == 0) atomicExch(p.status, 1);      // a load never completed
		const unsigned long long t0 = global_timer_ns();          // copies in flight land before the CTA may end
		while (global_timer_ns() - t0 < 1000000ull) __nanosleep(1000);
	}
	choose(p, best, &s_last);
}

// Stages of the ring kernel for these sizes: 5 where the rows leave room; 0: it does not fit.
int ring_stages(const DenseArgs &a) {
	const long long room = 227 * 1024 - RG_STATIC - (long long)a.M * ((a.K + 63) / 64 * 128 + 16);
	const int n = room < 0 ? 0 : (int)std::min<long long>(RG_STAGES, room / (DN_WARPS * RG_BOX));
	return n >= 3 ? n : 0;
}

// Where the kernel with two CTAs per SM is the faster one all the same (us, that one / ring; `smem`: what its rows take).
//   Two K slices per warp on many tiles: the barrier and the sums of a tile outweigh its copies.  768 -> 32000 12.9 / 13.9, -> 64000 22.9 / 26.3, 576 -> 64000
//   20.8 / 25.3; on fewer tiles the other way round (768 -> 4768 4.4 / 3.8, 5 rows -> 8192 6.1 / 5.7, rows prepared here -> 16384 14.0 / 13.3); with a whole
//   multiple of slices 1024 -> 32000 14.9 / 14.6, -> 64000 26.6 / 28.2.  One slice
//   per warp (512 -> 64000 .91) and three (1280 .92) are not affected, four uneven ones (1664 -> 64000 43.0 / 44.0) a little.
//   Long rows, where a tile takes as long as the launch, and tiles that fill as many rounds here as half rounds there: 8192 -> 7136 25.1 / 27.1, -> 2400 12.8 / 13.3,
//   -> 12240 37.4 / 38.9; with one round less the ring wins (-> 4768 .88, -> 9504 .96), and so it does where the rows leave room for one CTA only or for
//   little L1 beside two (5 rows .75).
bool ring_loses(const DenseArgs &a, int ntiles, size_t smem) {
	const int units = (a.K + 63) >> 6, sms = dn_sm_count();
	if (units > 8 && units <= 16) return ntiles > (units == 16 ? 2048 : a.prep ? 1280 : 640);
	if (units > 24 && units < 32) return ntiles > 1536;
	return a.K >= 8192 && smem <= 68 * 1024 && !(a.prep && ntiles <= 2 * sms) && (ntiles + sms - 1) / sms == 2 * ((ntiles + 2 * sms - 1) / (2 * sms));
}

int launch_ring(const DenseArgs &a, int stages, cudaStream_t stream) {
	alignas(64) CUtensorMap tmw;
	if (int rc = dense_tensor_map(a.w, a.N, a.K, a.ldw, 16, 64, &tmw)) return rc;
	const size_t smem = std::max((size_t)RG_MIN_SMEM, (size_t)DN_WARPS * stages * RG_BOX + (size_t)a.M * ((a.K + 63) / 64 * 128 + 16));
	// (the carve-out that it uses: the launches behind it keep the rest as L1; 259 -> 251 us per step of the state-space model)
	return dn_launch_as(1, (int)((smem + RG_STATIC) * 100 / (228 * 1024)) + 1, dense_ring_kernel, dim3(std::min((a.N + 15) / 16, dn_sm_count())), dim3(DN_THREADS), smem, stream, tmw, a, stages);
}

template <typename T>
int launch(const DenseArgs &a, cudaStream_t stream) {
	const size_t smem = (size_t)a.M * ((size_t)a.K * sizeof(T) + 16);
	const int ntiles = (a.N + 15) / 16, slots = dn_sm_count() * (smem + SK_STATIC > 110 * 1024 ? 1 : 2);
	// few tiles with long rows: a cluster per tile, as long as every warp of it has a step of K (with shorter rows the launch of a
	// cluster costs more than it saves)
	int kparts = a.K * (int)sizeof(T) > 8192 ? SK_PARTS : 1;
	while (kparts > 1 && (ntiles * kparts > dn_sm_count() || a.K < kparts * DN_WARPS * 64 / (int)sizeof(T))) kparts >>= 1;
	if (kparts > 1 && !a.e.best && smem <= 160 * 1024) return dn_launch_as(kparts, -1, dense_skinny_kernel<T, true>, dim3(ntiles * kparts), dim3(DN_THREADS), smem, stream, a, kparts);
	// Up to five rows: per decode step of a latent-attention model in us, this kernel / the one below: 8 layers of 2048 hidden, 1 row 381 / 433; 4 and
	// 3 layers of 2048 and 4096, 2 rows 228 / 251 and 358 / 361, 5 rows 279 / 294 and 397 / 421; 8 rows 297 / 341 and 486 / 472 (there the rows
	// of the widest layers do not fit, and every change between the two kernels' shared-memory splits costs more than the kernel gains).
	if (sizeof(T) == 2 && a.M <= RG_ROWS && !ring_loses(a, ntiles, smem))
		if (const int stages = ring_stages(a)) return launch_ring(a, stages, stream);
	const int waves = (ntiles + slots - 1) / slots;
	return dn_launch(dense_skinny_kernel<T, false>, dim3((ntiles + waves - 1) / waves), dim3(DN_THREADS), smem, stream, a, 1);
}

}   // namespace

bool dense_skinny_ok(int M, int K, int dtype) { return M >= 1 && M <= SK_M && (size_t)M * ((size_t)K * (dtype ? 4 : 2) + 16) <= SK_SMEM_MAX; }

int dense_skinny_launch(const DenseArgs &a, int dtype, cudaStream_t stream) {
	return dtype ? launch<float>(a, stream) : launch<bf16>(a, stream);
}

// ---- the same row preparation as a kernel of its own (prompts, and many rows) -------------------------------------------
template <typename T>
__global__ void __launch_bounds__(DN_THREADS) dense_rows_kernel(const RowPrep p, T *h, long long ldh) {
	__shared__ float s_norm[RP_SMEM];
	pdl_wait();
	pdl_trigger();
	prepare_row<T>(p, blockIdx.x, h + (size_t)blockIdx.x * ldh, p.x_out != nullptr, s_norm);
}

int dense_rows_launch(const RowPrep &p, int M, void *h, long long ldh, int dtype, cudaStream_t stream) {
	if (dtype) return dn_launch(dense_rows_kernel<float>, dim3(M), dim3(DN_THREADS), 0, stream, p, reinterpret_cast<float *>(h), ldh);
	return dn_launch(dense_rows_kernel<bf16>, dim3(M), dim3(DN_THREADS), 0, stream, p, reinterpret_cast<bf16 *>(h), ldh);
}

}   // namespace gptq
