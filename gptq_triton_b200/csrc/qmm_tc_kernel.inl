// Body of the tcgen05 prefill kernel; included by qmm_tc.cu.
namespace gptq {

// KP: K-blocks of 64 per stage.  Two halve the waits, arrivals and commits per K-block, which compete with the dequantisation for issue
// slots; one lets four stages of 256 rows fit.
template <int EPI, int KP>
__global__ void __launch_bounds__(TC_THREADS, 1) tc_kernel(const __grid_constant__ CUtensorMap tmx, const __grid_constant__ CUtensorMap tmw0,
														   const __grid_constant__ CUtensorMap tmw1, const TcParams p) {
	extern __shared__ __align__(1024) unsigned char smem[];
	constexpr bool PAIR = (EPI == TC_EPI_SILU);              // 64 gate and 64 up columns per tile
	constexpr int TN = PAIR ? 64 : 128;                      // columns of a weight tensor per tile
	const TcArgs &a = p.a;
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	const int m0 = blockIdx.x * p.nr, n0 = blockIdx.y * TN;
	const int split = blockIdx.z, splits = gridDim.z;
	const int kb0 = split * p.kb_per_split, nkb = min(p.kb_per_split, a.K / TC_BK - kb0);
	const int n = (nkb + KP - 1) / KP, S = p.s_stages, PW = p.w_stages;
	constexpr int W_SC = TC_W_SC(KP), W_QZ = TC_W_QZ(KP), W_STAGE = TC_W_STAGE(KP);
	const int sets = a.groupsize % (KP * TC_BK) ? KP : 1;      // the halves of a stage may lie in different groups
	const uint32_t x_block = (uint32_t)p.nr * (TC_BK * 2), x_stage = x_block * KP;

	// shared memory: [X ring | packed-weight ring | barriers]; the X ring becomes the epilogue's fp32 tile [nr][128]
	const uint32_t sX = smem_u32(smem), sW = sX + S * x_stage;
	uint64_t *bars = reinterpret_cast<uint64_t *>(smem + p.bar_off);
	const uint32_t bar_full = smem_u32(bars), bar_empty = bar_full + 8 * TC_MAX_STAGES;
	const uint32_t bar_full_w = bar_empty + 8 * TC_MAX_STAGES, bar_empty_w = bar_full_w + 8 * TC_MAX_WSTAGES;
	const uint32_t bar_acc = bar_empty_w + 8 * TC_MAX_WSTAGES;
	uint32_t *s_tmem = reinterpret_cast<uint32_t *>(bars + TC_BARS);
	volatile int *s_abort = reinterpret_cast<volatile int *>(s_tmem + 1);

	if (tid == 0) {
		for (int s = 0; s < S; ++s) {
			mbar_init(bar_full + 8 * s, 5);                   // four dequantise warps and the X producer
			mbar_init(bar_empty + 8 * s, 1);
		}
		for (int s = 0; s < PW; ++s) {
			mbar_init(bar_full_w + 8 * s, 2);                 // words; scales and zeros
			mbar_init(bar_empty_w + 8 * s, 4);                // one arrival per warp of the consuming group
		}
		mbar_init(bar_acc, 1);
		*s_abort = 0;
		fence_mbar_init();
		tma_prefetch_desc(&tmx);
		tma_prefetch_desc(&tmw0);
		if (PAIR) tma_prefetch_desc(&tmw1);
	}
	if (warp == 3) {
		tmem_alloc(smem_u32(s_tmem), TC_TMEM_COLS);
		tmem_relinquish();
	}
	tc_fence_before();
	__syncthreads();
	tc_fence_after();
	const uint32_t tmem = *s_tmem, tmem_a = tmem + TC_TMEM_COLS - S * (KP * TC_BK / 2);      // accumulators in front

	pdl_wait();          // nothing of earlier kernels, weights included, has been touched so far

	auto fail = [&]() {
		*s_abort = 1;
		atomicExch(p.status, 3);           // 3: a wait inside the tensor-core kernel ran out
	};
	// a producer that gives up leaves its copies a millisecond to land before the CTA may end
	auto settle = [&]() {
		const unsigned long long t0 = global_timer_ns();
		while (global_timer_ns() - t0 < 1000000ull) __nanosleep(1000);
	};

	// One lane of the three serial roles does the work, but the whole warp walks the loop: its addresses and descriptors are then
	// warp-uniform.  With a loop for lane 0 alone the issuer needed 0.40 us per K-block and was the bound of every short prompt
	// (M = 40, 4096 -> 12288: 28.3 us; uniform: 16.4 us; with two K-blocks per stage 13.9 us).
	if (warp == 0 || warp == 3) {
		// ---------------- packed weights (warp 0), scales and zeros (warp 3) ----------------
		const int gk = a.groupsize / TC_BK, nz = a.N >> 3, g0 = kb0 / gk;
		int left = gk - (kb0 - g0 * gk), s = 0, row = kb0 * 8, groups = a.K / a.groupsize - g0;      // blocks left in the group, groups left
		const __half *sc0 = a.sc0 + (size_t)g0 * a.N + n0, *sc1 = PAIR ? a.sc1 + (size_t)g0 * a.N + n0 : nullptr;
		const int32_t *qz0 = a.qz0 + (size_t)g0 * nz + (n0 >> 3), *qz1 = PAIR ? a.qz1 + (size_t)g0 * nz + (n0 >> 3) : nullptr;
		uint32_t ph = 1, dst = sW, bar = bar_full_w;
		const bool one = tc_elect();
		for (int i = 0; i < n; ++i) {
			if (!tc_wait(bar + (bar_empty_w - bar_full_w), ph, s_abort)) { fail(); settle(); break; }
			if (one) {
				if (warp == 0) {
					mbar_arrive_expect_tx(bar, W_SC);
					tma_load_2d(dst, &tmw0, n0, row, bar);             // (packed rows behind K read as zero)
					if (PAIR) tma_load_2d(dst + W_SC / 2, &tmw1, n0, row, bar);
				} else {
					auto group = [&](int h, size_t more) {
						const uint32_t sc = dst + W_SC + h * 256, qz = dst + W_QZ + h * 64;
						tc_bulk_load(sc, sc0 + more * a.N, TN * 2, bar);
						tc_bulk_load(qz, qz0 + more * nz, TN / 2, bar);
						if (PAIR) {
							tc_bulk_load(sc + 128, sc1 + more * a.N, TN * 2, bar);
							tc_bulk_load(qz + 32, qz1 + more * nz, TN / 2, bar);
						}
					};
					mbar_arrive_expect_tx(bar, sets * 320);
					group(0, 0);
					if (KP == 2 && sets == 2) group(1, left == 1 && groups > 1 ? 1 : 0);
				}
			}
			__syncwarp();
			row += 8 * KP;
#pragma unroll
			for (int h = 0; h < KP; ++h)
				if (--left == 0) {
					left = gk;
					--groups;
					sc0 += a.N;
					qz0 += nz;
					if (PAIR) {
						sc1 += a.N;
						qz1 += nz;
					}
				}
			dst += W_STAGE;
			bar += 8;
			if (++s == PW) {
				s = 0;
				dst = sW;
				bar = bar_full_w;
				ph ^= 1;
			}
		}
	} else if (warp == 1) {
		// ---------------- X tiles (rows beyond M and columns beyond K are filled with zeros by the copy) ----------------
		int s = 0;
		uint32_t ph = 1;
		const bool one = tc_elect();
		for (int i = 0; i < n; ++i) {
			if (!tc_wait(bar_empty + 8 * s, ph, s_abort)) { fail(); settle(); break; }
			if (one) {
				mbar_arrive_expect_tx(bar_full + 8 * s, x_stage);
#pragma unroll
				for (int h = 0; h < KP; ++h) tma_load_2d(sX + s * x_stage + h * x_block, &tmx, (kb0 + KP * i + h) * TC_BK, m0, bar_full + 8 * s);
			}
			__syncwarp();
			if (++s == S) {
				s = 0;
				ph ^= 1;
			}
		}
	} else if (warp == 2) {
		// ---------------- MMA issuer ----------------
		const uint32_t idesc = (1u << 4) | ((uint32_t)(p.nr >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);   // D fp32, A/B fp16 K-major, N = nr, M = 128
		uint64_t xd = smem_desc_sw128(sX);
		uint32_t at = tmem_a, ph = 0, acc = 0, bar = bar_full;
		const uint32_t bar_end = bar_full + 8 * S;
		const bool one = tc_elect();
		for (int i = 0; i < n; ++i) {
			if (!tc_wait(bar, ph, s_abort)) { fail(); break; }
			tc_fence_after();
			if (one) {
				// (where K ends on an odd block, the second block of the last stage is zero in X and in the weights)
#pragma unroll
				for (int k = 0; k < KP * TC_BK / 16; ++k)
					umma_f16_ts(tmem, at + 8 * k, xd + (uint64_t)((k >> 2) * (x_block >> 4) + 2 * (k & 3)), idesc, k == 0 ? acc : 1u);
				umma_commit(bar + (bar_empty - bar_full));          // stage free once these MMAs have read it
			}
			__syncwarp();
			acc = 1;
			xd += x_stage >> 4;
			at += KP * TC_BK / 2;
			bar += 8;
			if (bar == bar_end) {
				bar = bar_full;
				xd -= (uint64_t)(S * (x_stage >> 4));
				at = tmem_a;
				ph ^= 1;
			}
		}
		if (one) umma_commit(bar_acc);                   // accumulators complete
		__syncwarp();
	} else if (warp >= 4) {
		// ---------------- dequantise: group j takes the stages j, j + 4, ... ----------------
		// A stage's empty barrier is never two phases away from its waiter: a group is at most S >= 4 stages ahead of the MMAs.
		// A stage of the packed ring is always read by the same group (PW is a multiple of 4).
		const int q = warp & 3, grp = (warp - 4) >> 2, wt = q * 32 + lane;      // tensor-memory lane = weight column of the tile
		const uint32_t w_off = PAIR ? (uint32_t)((wt >> 6) * (W_SC / 2) + (wt & 63) * 4) : (uint32_t)(wt * 4);
		constexpr uint32_t W_ROW = PAIR ? 256 : 512;
		const uint32_t zsh = (wt & 7) * 4, a_dst = tmem_a + ((uint32_t)(q * 32) << 16);
		int s = grp;
		uint32_t st = sW + grp * W_STAGE, w_bar = bar_full_w + 8 * grp, wp = 0, sp = 1;
		const uint32_t st_end = sW + PW * W_STAGE;
		bool ok = true;
		for (int i = grp; i < n; i += TC_GROUPS) {
			ok = tc_wait_inline(w_bar, wp, s_abort) && tc_wait_inline(bar_empty + 8 * s, sp, s_abort);      // the whole warp goes on or none of it
			if (!ok) break;
			tc_fence_after();
			uint32_t sc, ze, zo;
			auto weights = [&](int h, uint32_t(&o)[32]) {
				uint32_t w[8];
#pragma unroll
				for (int r = 0; r < 8; ++r) w[r] = tc_lds32(st + w_off + (8 * h + r) * W_ROW);
				if (h == 0 || sets == 2) {
					sc = tc_lds16(st + W_SC + h * 256 + wt * 2) * 0x00010001u;
					// behind an odd number of K-blocks: exact zeros.  (0 - zero) * scale may be infinite in fp16, times the zeros of X a NaN
					if (KP == 2 && h == 1 && 2 * i + 1 >= nkb) sc = 0u;
					const uint32_t zz = ((tc_lds32(st + W_QZ + h * 64 + (wt >> 3) * 4) >> zsh) & 0xFu) + 1u;
					ze = (0x6400u + zz) * 0x00010001u;            // half2(1024 + zero)
					zo = (0xD400u + (zz << 4)) * 0x00010001u;     // half2(-(64 + zero))
				}
#pragma unroll
				for (int r = 0; r < 8; ++r) {
					const uint32_t w8 = w[r] >> 8;
					const uint32_t p04 = h2_mul(h2_sub(lop3_and_or(w[r], MASK_LO, MAGIC_1024), ze), sc);
					const uint32_t p15 = h2_mul(h2_fma(lop3_and_or(w[r], MASK_HI, MAGIC_1024), 0x2C002C00u, zo), sc);
					const uint32_t p26 = h2_mul(h2_sub(lop3_and_or(w8, MASK_LO, MAGIC_1024), ze), sc);
					const uint32_t p37 = h2_mul(h2_fma(lop3_and_or(w8, MASK_HI, MAGIC_1024), 0x2C002C00u, zo), sc);
					o[4 * r] = __byte_perm(p04, p15, 0x5410);                // natural k order k0 .. k7
					o[4 * r + 1] = __byte_perm(p26, p37, 0x5410);
					o[4 * r + 2] = __byte_perm(p04, p15, 0x7632);
					o[4 * r + 3] = __byte_perm(p26, p37, 0x7632);
				}
			};
#pragma unroll
			for (int h = 0; h < KP; ++h) {
				uint32_t o[32];
				weights(h, o);
				if (h == KP - 1) {
					__syncwarp();
					if (lane == 0) mbar_arrive(w_bar + (bar_empty_w - bar_full_w));
				}
				tmem_st32(a_dst + (s * KP + h) * (TC_BK / 2), o);
			}
			tmem_st_wait();
			tc_fence_before();
			__syncwarp();
			if (lane == 0) mbar_arrive(bar_full + 8 * s);
			s += TC_GROUPS;
			if (s >= S) {
				s -= S;
				sp ^= 1;
			}
			st += TC_GROUPS * W_STAGE;
			w_bar += TC_GROUPS * 8;
			if (st >= st_end) {
				st = sW + grp * W_STAGE;
				w_bar = bar_full_w + 8 * grp;
				wp ^= 1;
			}
		}
		if (!ok) fail();
		__syncwarp();

		// ---------------- accumulators [column][row] -> fp32 tile [row][128] over the drained X ring ----------------
		if (__all_sync(0xffffffffu, mbar_wait_bounded(bar_acc, 0, TC_SPIN))) {
			tc_fence_after();
			float *tile = reinterpret_cast<float *>(smem);
#pragma unroll 1
			for (int c = grp * 16; c < p.nr; c += 64) {
				float v[16];
				tmem_ld16(tmem + c + ((uint32_t)(q * 32) << 16), v);
				tmem_ld_wait();
#pragma unroll
				for (int j = 0; j < 16; ++j) tile[(c + j) * 128 + wt] = v[j];
			}
		} else {
			fail();
		}
		tc_fence_before();
	}
	if (splits > 1) tc_cluster_sync();
	else __syncthreads();
	if (warp == 3) {
		// tensor memory goes back only after every MMA issued above has completed (also when unwinding)
		if (lane == 0) mbar_wait_bounded(bar_acc, 0, TC_SPIN);
		__syncwarp();
		tc_fence_after();
		tmem_dealloc(tmem, TC_TMEM_COLS);
	}

	// ---------------- epilogue: the CTAs of a split share the rows; partial tiles are summed in split order ----------------
	const int live = min(p.nr, a.M - m0);
	const int rows = (live - split + splits - 1) / splits;          // rows split, split + splits, ...
	auto gather = [&](int row, int col) -> float4 {
		const uint32_t at = sX + (uint32_t)(row * 128 + col) * 4;
		if (splits == 1) return tc_lds128(at);
		float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
		float4 v[8];
#pragma unroll
		for (int i = 0; i < 8; ++i)
			if (i < splits) v[i] = tc_ld_peer(at, i);
#pragma unroll
		for (int i = 0; i < 8; ++i)
			if (i < splits) {
				r.x += v[i].x;
				r.y += v[i].y;
				r.z += v[i].z;
				r.w += v[i].w;
			}
		return r;
	};
	auto pack = [](float x, float y, float z, float w) {
		const __half2 lo = __floats2half2_rn(x, y), hi = __floats2half2_rn(z, w);
		return make_uint2(*reinterpret_cast<const uint32_t *>(&lo), *reinterpret_cast<const uint32_t *>(&hi));
	};
	auto add4 = [](float4 &v, const __half *src) {
		const uint2 u = *reinterpret_cast<const uint2 *>(src);
		const float2 lo = __half22float2(*reinterpret_cast<const __half2 *>(&u.x)), hi = __half22float2(*reinterpret_cast<const __half2 *>(&u.y));
		v.x += lo.x;
		v.y += lo.y;
		v.z += hi.x;
		v.w += hi.y;
	};
	if (EPI == TC_EPI_PLAIN) {
#pragma unroll 2
		for (int e = tid; e < rows * 32; e += TC_THREADS) {
			const int row = split + (e >> 5) * splits, col = (e & 31) * 4;
			float4 v = gather(row, col);
			if (a.bias) add4(v, a.bias + n0 + col);
			if (a.residual) add4(v, a.residual + (size_t)(m0 + row) * a.ldr + n0 + col);
			*reinterpret_cast<uint2 *>(a.y + (size_t)(m0 + row) * a.ldy + n0 + col) = pack(v.x, v.y, v.z, v.w);
		}
	} else if (EPI == TC_EPI_SILU) {
#pragma unroll 2
		for (int e = tid; e < rows * 16; e += TC_THREADS) {
			const int row = split + (e >> 4) * splits, col = (e & 15) * 4;
			const float4 v = gather(row, col), u = gather(row, col + 64);
			*reinterpret_cast<uint2 *>(a.y + (size_t)(m0 + row) * a.ldy + n0 + col) =
				pack(silu_f32(v.x) * u.x, silu_f32(v.y) * u.y, silu_f32(v.z) * u.z, silu_f32(v.w) * u.w);
		}
	} else {
		// the tile is one head of section Q, K or V
		const int section = n0 / a.hidden, head = (n0 - section * a.hidden) >> 7;
#pragma unroll 1
		for (int e = tid; e < rows * 16; e += TC_THREADS) {
			const int row = m0 + split + (e >> 4) * splits, d = (e & 15) * 4;
			int pos = a.pos[row];
			if (pos < 0 || pos >= a.max_pos) {      // never index the tables / the cache out of range
				atomicExch(p.status, 4);
				if (section != 0) continue;         // K / V of such a row are dropped, not written over cache row 0
				pos = 0;
			}
			const float4 x1 = gather(row - m0, d), x2 = gather(row - m0, d + 64);
			float lo[4] = {x1.x, x1.y, x1.z, x1.w}, hi[4] = {x2.x, x2.y, x2.z, x2.w};
			if (section < 2) {
				const __half *ct = a.cos_t + (size_t)pos * 128 + d, *st = a.sin_t + (size_t)pos * 128 + d;
#pragma unroll
				for (int i = 0; i < 4; ++i) {
					const float u = lo[i], v = hi[i];
					lo[i] = u * __half2float(ct[i]) - v * __half2float(st[i]);
					hi[i] = v * __half2float(ct[i + 64]) + u * __half2float(st[i + 64]);
				}
			}
			__half *dst;
			if (section == 0) {
				dst = a.q_out + (size_t)row * a.q_stride_m + head * 128;
			} else {
				const int bi = row / a.tokens_per_batch, ti = row - bi * a.tokens_per_batch;
				dst = (section == 1 ? a.k_out : a.v_out) + (size_t)bi * a.kv_sb + (size_t)ti * a.kv_st + (size_t)head * a.kv_sh + (size_t)pos * a.kv_sp;
			}
			const uint2 l = pack(lo[0], lo[1], lo[2], lo[3]), h = pack(hi[0], hi[1], hi[2], hi[3]);
			if (p.out8) {
				*reinterpret_cast<uint2 *>(dst + d) = l;
				*reinterpret_cast<uint2 *>(dst + d + 64) = h;
			} else {
				*reinterpret_cast<uint32_t *>(dst + d) = l.x;
				*reinterpret_cast<uint32_t *>(dst + d + 2) = l.y;
				*reinterpret_cast<uint32_t *>(dst + d + 64) = h.x;
				*reinterpret_cast<uint32_t *>(dst + d + 66) = h.y;
			}
		}
	}
	if (splits > 1) tc_cluster_sync();          // the peers have read this CTA's tile
}

}   // namespace gptq
