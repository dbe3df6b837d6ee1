// What the kernels of the matrix-state recurrences share (seqmix.cu: token by token, chunked_recurrence.cu: in chunks).
#pragma once
#include "common.cuh"

__device__ __forceinline__ float softplus_f(float x) { return x > 20.f ? x : log1pf(expf(x)); }
__device__ __forceinline__ float silu_f(float x) { return x / (1.f + expf(-x)); }
// what a gate does to the projection it is made from: 0 sigmoid, 1 silu
__device__ __forceinline__ float gate_f(float x, int act) { const float s = 1.f / (1.f + expf(-x)); return act == 1 ? x * s : s; }
// where the decay of a token comes from: a projection per head and key channel, a projection per head, or a constant
// per head (`A_log` then holds the constants themselves and the recurrence is plain linear attention: q, k and v pass
// silu instead of the unit norms, and the state takes k v^T without the correction towards v)
// or (DECAY_FORGET_GATE) a forget gate per head and key channel that also decides what is written: with `a_in` the
// gate's projection, `dt_bias` its bias and `A_log` a lower bound per head and key channel, f = low + (1 - low) *
// sigmoid(a + bias), S <- diag(f) S + (1 - f) v^T, o = S^T silu(q): the key is 1 - f, there is no key projection (a
// row of `qkv` holds the queries and then the values), no unit norms and no correction towards v
// or (DECAY_LOG_SIGMOID) a gate per head and key channel raised to a power: with `a_in` the gate's projection, `dt_bias`
// its bias and `A_log` the power itself per head (1 / tau), g = sigmoid(a + bias)^power = exp(-power * softplus(-(a + bias))),
// S <- diag(g) S + k v^T, o = S^T (q * q_scale): gated linear attention, no unit norms, no correction
// or (DECAY_STEP) a step size per head and token: with `a_in` (n, H) its projection and `dt_bias` (H) its bias,
// dt = softplus(a + bias), S <- exp(-exp(A_log[head]) * dt) S + k (dt v)^T, o = S^T q: a selective state space in its
// recurrent form (k is the input matrix B, q the output matrix C, v the head's inputs); the outputs leave unnormalised
// or (DECAY_BONUS) a decay per head and key channel with a bonus for the current token: with `a_in` the decay's projection,
// `dt_bias` its bias and `A_log` the bonus u per head and key channel, g = exp(-exp(a + bias)), o = (S + diag(u) k v^T)^T q,
// then S <- diag(g) S + k v^T: the outputs read the state before the token.  The bonus' share of o is (sum_i u_i q_i k_i) v,
// one number a token (kept where the other forms keep beta).  The norm's weights are the head's own (H * v_dim of them)
enum { DECAY_PER_CHANNEL = 0, DECAY_PER_HEAD = 1, DECAY_CONSTANT = 2, DECAY_FORGET_GATE = 3, DECAY_LOG_SIGMOID = 4,
       DECAY_STEP = 5, DECAY_BONUS = 6 };

// What the kernels of the chunked form get (chunked_recurrence.cu): the first `segments` of the `all_segments` requests of a
// step of `all_rows` rows, n rows at most.  Scratch arrays are indexed by (chunk, head), but for
//   again    (segment, head): 0, or 1 + the first chunk of a portion that the walk has to take again, because numbers
//            that are not finite came up in it, from the state that `s` holds for that chunk
//   chunked  (last row of a request, head): whether its rows are the chunked form's
constexpr int REC_CHUNK = 64;
struct ChunkArgs {
    const void* qkv; int ld;
    const void* b_in; int ldb;
    const void* a_in; int lda;
    const void* gate; int ldg;
    const float *A_log, *dt_bias, *norm_w;
    float eps, unit_eps, q_scale;
    float* state; size_t state_stride;
    void* out; int ldo;
    float* o_raw;
    const int *row_slot, *row_last, *seg_row0;
    int segments, all_segments, n, all_rows, H, G, mode, gate_act, chunks;
    float *qb, *kd, *w, *u, *a, *s, *decay;
    int *again, *chunked;
};
// Whether the chunked kernels take these widths, and, if so, whether these operands: 16-byte rows and states.
bool chunked_recurrence_takes(int dtype, const ChunkArgs& args, int k_dim, int v_dim);
// Launches them (scratch: tis_chunked_recurrence_floats), and leaves the arrays in the scratch in `args`.
int chunked_recurrence(int dtype, ChunkArgs& args, int k_dim, int v_dim, float* scratch, size_t scratch_floats, cudaStream_t stream);
