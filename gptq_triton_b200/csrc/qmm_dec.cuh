// Decode-regime (M <= 16) quantised matmul on the tcgen05 tensor cores.
#pragma once

#include "tcgen05.cuh"

namespace gptq {

enum { DEC_EPI_PLAIN = 0, DEC_EPI_SILU = 1, DEC_EPI_ROPE = 2 };

struct DecArgs {
	const __half *x;
	long long ldx;
	const int32_t *qw0, *qw1;
	const int32_t *qz0, *qz1;
	const __half *sc0, *sc1;
	int M, K, N, groupsize;
	// PLAIN / SILU
	const __half *bias, *residual;
	long long ldr;
	__half *y;
	long long ldy;
	float *ss_out;               // PLAIN: sums of squares of the outputs per 32 columns, or NULL
	// ROPE
	const __half *cos_t, *sin_t;
	const int32_t *pos;
	__half *q_out, *k_out, *v_out;
	long long q_stride_m, kv_sb, kv_st, kv_sh, kv_sp;
	int tokens_per_batch, hidden, max_pos;
};

bool dec_shape_ok(int M, int K, int N, int groupsize);
size_t dec_ws_bytes(int M);                              // arrival flags (the counter area, left zero) and partial sums
int dec_launch(const DecArgs &a, int epi, void *workspace, size_t ws_bytes, cudaStream_t stream);

}   // namespace gptq
