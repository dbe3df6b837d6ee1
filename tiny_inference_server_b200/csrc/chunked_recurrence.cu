// The matrix-state recurrences (recurrence.cuh) over long portions, REC_CHUNK tokens at a time.
//
//   S_t = diag(g_t) S_{t-1} + k_t u_t^T,   o_t = S_t^T q_t   (with a bonus: S_{t-1} and the token's own share)
//   u_t = c_t v_t, or for the delta rule u_t = beta_t (v_t - (diag(g_t) S_{t-1})^T k_t)
//
// Token by token this is a chain as long as the prompt with heads * v_dim independent columns.  Inside a chunk, with
// P(s, t] the product of the decays of tokens s+1..t per key channel and S_0 the state before the chunk,
//
//   o_t = (q_t P(0, t])^T S_0 + sum_{s <= t} A[t, s] u_s,      A[t, s] = sum_i q_ti k_si P(s, t]_i
//   S_C = diag(P(0, C]) S_0 + sum_s (k_s P(s, C]) u_s^T
//   delta rule: (I + diag(beta) L) U = diag(beta) V - diag(beta) (K P(0, .]) S_0,   L[t, s] = sum_i k_ti k_si P(s, t]_i (s < t)
//
// so everything but the state's way from chunk to chunk is independent of the other chunks, and dense:
//   chunk_prepare_kernel  a CTA per (chunk, head): the token vectors, A, and the chunk's share of the state
//                         (delta rule: the triangular system is solved for its two right sides, U = U0 - W S_0)
//   chunk_state_kernel    the states in front of the chunks: one multiply-add per element and chunk
//   chunk_delta_kernel    the same for the delta rule, whose U needs S_0: two products a chunk, a CTA per (16 columns, head)
//   chunk_output_kernel   a CTA per (chunk, head): [q P | A] [S_0; U], the norm over v_dim and the gate
//
// Every product of decays is a product of factors <= 1 in the direction the tokens run (within sub-chunks of 16 tokens,
// over whole sub-chunks between them): nothing is divided by a decay, so a decay of zero and a long product that
// underflows are what they are in the walk.  No token's output meets a later token's vectors, not even times zero.
// Everything is 32-bit (CUDA cores: 3 x tf32 on mma.sync measured 266 / 3 TFLOP/s against 67 here, and would have to
// split its operands first).
#include "recurrence.cuh"

namespace {

constexpr int C = REC_CHUNK, SUB = 16, NSUB = C / SUB;
constexpr int DCOLS = 16;                       // columns of the state that a CTA of chunk_delta_kernel takes

__device__ __forceinline__ void copy16(float* smem, const float* gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem));
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N> __device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// N neighbouring elements (2, 4) as floats; the address is a multiple of their size
template <int N> __device__ __forceinline__ void load_run(const float* p, float (&v)[N]) {
    if constexpr (N == 4) {
        const float4 x = *reinterpret_cast<const float4*>(p);
        v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
    } else {
        const float2 x = *reinterpret_cast<const float2*>(p);
        v[0] = x.x; v[1] = x.y;
    }
}
template <int N> __device__ __forceinline__ void load_run(const bf16* p, float (&v)[N]) {
    unsigned w[N / 2];
    if constexpr (N == 4) {
        const uint2 x = *reinterpret_cast<const uint2*>(p);
        w[0] = x.x; w[1] = x.y;
    } else {
        w[0] = *reinterpret_cast<const unsigned*>(p);
    }
#pragma unroll
    for (int i = 0; i < N / 2; ++i) {
        v[2 * i] = __uint_as_float(w[i] << 16);
        v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
}
template <int N> __device__ __forceinline__ void store_run(float* p, const float (&v)[N]) {
    if constexpr (N == 4) *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    else *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
}
template <int N> __device__ __forceinline__ void store_run(bf16* p, const float (&v)[N]) {
    __nv_bfloat162 h[N / 2];
#pragma unroll
    for (int i = 0; i < N / 2; ++i) h[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
    if constexpr (N == 4) *reinterpret_cast<uint2*>(p) = *reinterpret_cast<uint2*>(h);
    else *reinterpret_cast<__nv_bfloat162*>(p) = h[0];
}

// The rows of segment `seg`, 0 if it is padding or goes on where the one before it ended.
__device__ __forceinline__ int segment_rows(const ChunkArgs& p, int seg, int& row0) {
    row0 = p.seg_row0[seg];
    const int slot = p.row_slot[row0];
    if (slot < 0 || (row0 > 0 && p.row_slot[row0 - 1] == slot)) return 0;
    return p.row_last[row0] - row0 + 1;
}
// Where chunk `chunk` of the step lies (all lanes of a warp together): its first row and number of rows; false: there is
// no such chunk (the grid is sized by an upper bound).
__device__ __forceinline__ bool find_chunk(const ChunkArgs& p, int chunk, int& row0, int& rows) {
    const int lane = threadIdx.x & 31;
    int before = 0;
    for (int s0 = 0; s0 < p.segments; s0 += 32) {
        int first = 0, count = 0;
        if (s0 + lane < p.segments) count = segment_rows(p, s0 + lane, first);
        const int mine = (count + C - 1) / C;
        int upto = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += v;
        }
        const unsigned past = __ballot_sync(0xffffffffu, before + upto > chunk);
        if (past) {
            const int at = __ffs(past) - 1;
            const int in_segment = chunk - before - __shfl_sync(0xffffffffu, upto - mine, at);
            row0 = __shfl_sync(0xffffffffu, first, at) + in_segment * C;
            rows = min(C, __shfl_sync(0xffffffffu, count, at) - in_segment * C);
            return true;
        }
        before += __shfl_sync(0xffffffffu, upto, 31);
    }
    return false;
}
// The first chunk of segment `seg`, and its rows (all lanes of a warp together).
__device__ __forceinline__ int first_chunk(const ChunkArgs& p, int seg, int& row0, int& rows) {
    const int lane = threadIdx.x & 31;
    int before = 0, first;
    for (int s = lane; s < seg; s += 32) before += (segment_rows(p, s, first) + C - 1) / C;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
    rows = segment_rows(p, seg, row0);
    return before;
}

template <int K> struct PrepareSmem {
    static constexpr int ROW = K + 4;                       // padding: neighbouring tokens lie four banks apart
    static constexpr size_t bytes(bool delta) {
        return sizeof(float) * (3 * (size_t)C * ROW + NSUB * K + C + (delta ? SUB * SUB * NSUB * (NSUB + 1) / 2 : 0));
    }
};

// Bound by the issue of shared-memory loads and multiply-adds (1.5 M multiply-adds a chunk and head of 128 x 128, two CTAs
// an SM).  Blocks of A and L on the diagonal (16 x 16 tokens) are walked with a running key, P(s, t] k_s, so that they
// need neither divisions nor exponentials; the others factor at the sub-chunk edges.
template <typename T, int K, int V, bool DELTA>
__global__ void __launch_bounds__(256, 2) chunk_prepare_kernel(const ChunkArgs p) {
    constexpr int ROW = PrepareSmem<K>::ROW, CPL = K / 32;
    extern __shared__ __align__(16) float smem[];
    float* qs = smem;                                       // [C][ROW]  q, then q P(start of its sub-chunk, t]
    float* ks = qs + C * ROW;                               // k, then the same product
    float* gs = ks + C * ROW;                               // decays, then k P(t, end of its sub-chunk]
    float* subp = gs + C * ROW;                             // [NSUB][K] decay of a whole sub-chunk
    float* betas = subp + NSUB * K;                         // [C]
    float* M = betas + C;                                   // diag(beta) L, sub-chunk a's rows 16 (a + 1) long
    pdl_launch_dependents();
    const int head = blockIdx.x, chunk = blockIdx.y;
    int row0, rows;
    if (!find_chunk(p, chunk, row0, rows)) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int kvh = head / (p.H / p.G), mode = p.mode;
    const bool forget = mode == DECAY_FORGET_GATE, plain = mode == DECAY_CONSTANT, bonus = mode == DECAY_BONUS;
    const bool per_head = mode == DECAY_PER_HEAD || mode == DECAY_STEP;
    const T* qkv = (const T*)p.qkv;
    const T* a_in = (const T*)p.a_in;
    const int q_off = kvh * K, k_off = p.G * K + kvh * K, v_off = (forget ? 1 : 2) * p.G * K + head * V;
    const float rate = (plain || mode == DECAY_LOG_SIGMOID) ? p.A_log[head] : ((forget || bonus) ? 0.f : expf(p.A_log[head]));
    const int ch0 = lane * CPL;
    float bias[CPL], low[CPL];
#pragma unroll
    for (int i = 0; i < CPL; ++i) {
        bias[i] = plain ? 0.f : p.dt_bias[per_head ? head : head * K + ch0 + i];
        low[i] = (forget || bonus) ? p.A_log[head * K + ch0 + i] : 0.f;
    }
    pdl_wait();
    // ---- the chunk's token vectors: a warp a token; tokens behind the end change nothing (k 0, decay 1)
#pragma unroll 4
    for (int t = warp; t < C; t += 8) {
        float q[CPL], k[CPL], g[CPL], beta = 0.f;
#pragma unroll
        for (int i = 0; i < CPL; ++i) { q[i] = 0.f; k[i] = 0.f; g[i] = 1.f; }
        if (t < rows) {
            const size_t rr = (size_t)(row0 + t);
            float a[CPL];
            load_run<CPL>(qkv + rr * p.ld + q_off + ch0, q);
            if (!forget) load_run<CPL>(qkv + rr * p.ld + k_off + ch0, k);
            if (per_head) a[0] = to_f32(a_in[rr * p.lda + head]);
            else if (!plain) load_run<CPL>(a_in + rr * p.lda + (size_t)head * K + ch0, a);
            if (DELTA) {
                beta = 1.f / (1.f + expf(-to_f32(((const T*)p.b_in)[rr * p.ldb + head])));
                float sq = 0.f, sk = 0.f;
#pragma unroll
                for (int i = 0; i < CPL; ++i) { sq = fmaf(q[i], q[i], sq); sk = fmaf(k[i], k[i], sk); }
                sq = warp_sum(sq);
                sk = warp_sum(sk);
                const float fq = p.q_scale / sqrtf(sq + p.unit_eps), fk = 1.f / sqrtf(sk + p.unit_eps);
                const float whole = per_head ? expf(-rate * softplus_f(a[0] + bias[0])) : 0.f;
#pragma unroll
                for (int i = 0; i < CPL; ++i) {
                    q[i] *= fq;
                    k[i] *= fk;
                    g[i] = per_head ? whole : expf(-rate * softplus_f(a[i] + bias[i]));
                }
            } else if (plain) {
                beta = 1.f;
#pragma unroll
                for (int i = 0; i < CPL; ++i) { q[i] = silu_f(q[i]); k[i] = silu_f(k[i]); g[i] = rate; }
            } else if (forget) {
                beta = 1.f;
#pragma unroll
                for (int i = 0; i < CPL; ++i) {
                    const float open = 1.f / (1.f + expf(a[i] + bias[i]));      // 1 - sigmoid of the gate
                    q[i] = silu_f(q[i]);
                    k[i] = (1.f - low[i]) * open;
                    g[i] = low[i] + (1.f - low[i]) * (1.f - open);
                }
            } else if (bonus) {
#pragma unroll
                for (int i = 0; i < CPL; ++i) {
                    q[i] *= p.q_scale;
                    g[i] = expf(-expf(a[i] + bias[i]));
                    beta = fmaf(q[i] * low[i], k[i], beta);
                }
                beta = warp_sum(beta);
            } else {
                const bool stepped = mode == DECAY_STEP;
                beta = stepped ? softplus_f(a[0] + bias[0]) : 1.f;
                const float whole = stepped ? expf(-rate * beta) : 0.f;
#pragma unroll
                for (int i = 0; i < CPL; ++i) {
                    q[i] *= p.q_scale;
                    g[i] = stepped ? whole : expf(-rate * softplus_f(-(a[i] + bias[i])));
                }
            }
        }
        store_run<CPL>(qs + t * ROW + ch0, q);
        store_run<CPL>(ks + t * ROW + ch0, k);
        store_run<CPL>(gs + t * ROW + ch0, g);
        if (lane == 0) betas[t] = beta;
    }
    __syncthreads();
    const size_t unit = (size_t)chunk * p.H + head;
    float* A = p.a + unit * C * C;
    // ---- blocks on the diagonal: a thread per (token s, quarter of the channels), down the tokens t of its sub-chunk
    {
        const int slice = tid & 3, s = tid >> 2, a0 = s & ~(SUB - 1);
        float4 w[K / 16];
#pragma unroll
        for (int j = 0; j < K / 16; ++j) w[j] = *reinterpret_cast<const float4*>(ks + s * ROW + (j * 4 + slice) * 4);
#pragma unroll 1
        for (int t = a0; t < a0 + SUB; ++t) {
            const float* qt = qs + t * ROW + slice * 4;
            const float* kt = ks + t * ROW + slice * 4;
            const float* gt = gs + t * ROW + slice * 4;
            float da = 0.f, db = 0.f, la = 0.f, lb = 0.f;
            if (!bonus && t > s) {
#pragma unroll
                for (int j = 0; j < K / 16; ++j) {
                    const float4 g = *reinterpret_cast<const float4*>(gt + j * 16);
                    w[j].x *= g.x; w[j].y *= g.y; w[j].z *= g.z; w[j].w *= g.w;
                }
            }
#pragma unroll
            for (int j = 0; j < K / 16; ++j) {
                const float4 q = *reinterpret_cast<const float4*>(qt + j * 16);
                da = fmaf(q.x, w[j].x, fmaf(q.y, w[j].y, da));
                db = fmaf(q.z, w[j].z, fmaf(q.w, w[j].w, db));
                if (DELTA) {
                    const float4 k = *reinterpret_cast<const float4*>(kt + j * 16);
                    la = fmaf(k.x, w[j].x, fmaf(k.y, w[j].y, la));
                    lb = fmaf(k.z, w[j].z, fmaf(k.w, w[j].w, lb));
                }
            }
            if (bonus && t > s) {
#pragma unroll
                for (int j = 0; j < K / 16; ++j) {
                    const float4 g = *reinterpret_cast<const float4*>(gt + j * 16);
                    w[j].x *= g.x; w[j].y *= g.y; w[j].z *= g.z; w[j].w *= g.w;
                }
            }
            float d = da + db;
            d += __shfl_xor_sync(0xffffffffu, d, 1);
            d += __shfl_xor_sync(0xffffffffu, d, 2);
            if (slice == 0 && t >= s) A[t * C + s] = (bonus && t == s) ? betas[t] : d;
            if (DELTA) {
                float l = la + lb;
                l += __shfl_xor_sync(0xffffffffu, l, 1);
                l += __shfl_xor_sync(0xffffffffu, l, 2);
                const int sub = a0 / SUB;
                if (slice == 0 && t > s) M[SUB * SUB * sub * (sub + 1) / 2 + (t - a0) * SUB * (sub + 1) + s] = betas[t] * l;
            }
        }
    }
    __syncthreads();
    // ---- products of decays inside the sub-chunks
    for (int idx = tid; idx < K * NSUB; idx += 256) {
        const int ch = idx % K, sub = idx / K;
        float g[SUB], k[SUB], pre = 1.f;
#pragma unroll
        for (int r = 0; r < SUB; ++r) {
            const int at = (sub * SUB + r) * ROW + ch;
            g[r] = gs[at];
            k[r] = ks[at];
            if (!bonus) pre *= g[r];
            qs[at] *= pre;
            if (DELTA) ks[at] = k[r] * pre;
            if (bonus) pre *= g[r];
        }
        subp[sub * K + ch] = pre;
        float suf = 1.f;
#pragma unroll
        for (int r = SUB - 1; r >= 0; --r) {
            gs[(sub * SUB + r) * ROW + ch] = k[r] * suf;
            suf *= g[r];
        }
    }
    __syncthreads();
    // ---- blocks below the diagonal: a warp each, rows (lane / 4) + 8 i, columns (lane % 4) + 4 j
    if (warp < 6) {
        const int a = warp < 3 ? 3 : (warp < 5 ? 2 : 1), b = warp < 3 ? warp : (warp < 5 ? warp - 3 : 0);
        const int t0 = a * SUB + (lane >> 2), s0 = b * SUB + (lane & 3);
        float acc[2][4] = {}, accl[2][4] = {};
        for (int c = 0; c < K; c += 4) {
            float4 between = make_float4(1.f, 1.f, 1.f, 1.f);
            for (int m = b + 1; m < a; ++m) {
                const float4 d = *reinterpret_cast<const float4*>(subp + m * K + c);
                between.x *= d.x; between.y *= d.y; between.z *= d.z; between.w *= d.w;
            }
            float4 kv[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                kv[j] = *reinterpret_cast<const float4*>(gs + (s0 + 4 * j) * ROW + c);
                kv[j].x *= between.x; kv[j].y *= between.y; kv[j].z *= between.z; kv[j].w *= between.w;
            }
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const float4 q = *reinterpret_cast<const float4*>(qs + (t0 + 8 * i) * ROW + c);
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    acc[i][j] = fmaf(q.x, kv[j].x, fmaf(q.y, kv[j].y, fmaf(q.z, kv[j].z, fmaf(q.w, kv[j].w, acc[i][j]))));
                if (DELTA) {
                    const float4 k = *reinterpret_cast<const float4*>(ks + (t0 + 8 * i) * ROW + c);
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        accl[i][j] = fmaf(k.x, kv[j].x, fmaf(k.y, kv[j].y, fmaf(k.z, kv[j].z, fmaf(k.w, kv[j].w, accl[i][j]))));
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int t = t0 + 8 * i, s = s0 + 4 * j;
                A[t * C + s] = acc[i][j];
                if (DELTA) M[SUB * SUB * a * (a + 1) / 2 + (t - a * SUB) * SUB * (a + 1) + s] = betas[t] * accl[i][j];
            }
    }
    // ---- what the other kernels read: q P(0, t], the chunk's decay, k P(t, C]
    float* qb = p.qb + unit * C * K;
    for (int idx = tid; idx < K / 4 * C; idx += 256) {
        const int ch = idx % (K / 4) * 4, t = idx / (K / 4), sub = t / SUB;
        float4 q = *reinterpret_cast<const float4*>(qs + t * ROW + ch);
        for (int m = 0; m < sub; ++m) {
            const float4 d = *reinterpret_cast<const float4*>(subp + m * K + ch);
            q.x *= d.x; q.y *= d.y; q.z *= d.z; q.w *= d.w;
        }
        *reinterpret_cast<float4*>(qb + t * K + ch) = q;
    }
    for (int ch = tid; ch < K; ch += 256) {
        float d = 1.f;
#pragma unroll
        for (int m = 0; m < NSUB; ++m) d *= subp[m * K + ch];
        p.decay[unit * K + ch] = d;
    }
    float* ub = p.u + unit * C * V;
    __syncthreads();                                        // gs, qs and M are complete, nobody reads gs as it was
    if (DELTA) {
        float* kd = p.kd + unit * C * K;
        for (int idx = tid; idx < K / 4 * C; idx += 256) {
            const int ch = idx % (K / 4) * 4, t = idx / (K / 4), sub = t / SUB;
            float4 k = *reinterpret_cast<const float4*>(gs + t * ROW + ch);
            for (int m = sub + 1; m < NSUB; ++m) {
                const float4 d = *reinterpret_cast<const float4*>(subp + m * K + ch);
                k.x *= d.x; k.y *= d.y; k.z *= d.z; k.w *= d.w;
            }
            *reinterpret_cast<float4*>(kd + t * K + ch) = k;
        }
        // the triangular system, a thread a column of [beta K P(0, .] | beta V]
        for (int col = tid; col < K + V; col += 256) {
            float x[C];
            const bool key = col < K;
            if (key) {
                float pre = 1.f;
#pragma unroll
                for (int t = 0; t < C; ++t) {
                    if (t > 0 && t % SUB == 0) pre *= subp[(t / SUB - 1) * K + col];
                    x[t] = betas[t] * ks[t * ROW + col] * pre;
                }
            } else {
#pragma unroll
                for (int t = 0; t < C; ++t)
                    x[t] = t < rows ? betas[t] * to_f32(qkv[(size_t)(row0 + t) * p.ld + v_off + col - K]) : 0.f;
            }
            float* dst = key ? p.w + unit * C * K + col : ub + (col - K);
            const int ldd = key ? K : V;
#pragma unroll
            for (int t = 0; t < C; ++t) {
                const int sub = t / SUB;
                const float* m = M + SUB * SUB * sub * (sub + 1) / 2 + (t - sub * SUB) * SUB * (sub + 1);
                float y0 = x[t], y1 = 0.f;
#pragma unroll
                for (int s = 0; s + 3 < t; s += 4) {
                    const float4 v = *reinterpret_cast<const float4*>(m + s);
                    y0 = fmaf(-v.x, x[s], y0);
                    y1 = fmaf(-v.y, x[s + 1], y1);
                    y0 = fmaf(-v.z, x[s + 2], y0);
                    y1 = fmaf(-v.w, x[s + 3], y1);
                }
#pragma unroll
                for (int s = t & ~3; s < t; ++s) y0 = fmaf(-m[s], x[s], y0);
                x[t] = y0 + y1;
                dst[(size_t)t * ldd] = x[t];
            }
        }
        return;
    }
    // ---- the chunk's share of the state, sum_s (k_s P(s, C]) u_s^T: a thread 8 x 8 of it
    float* us = smem;                                       // [C][V], over the queries and keys
    for (int idx = tid; idx < K / 4 * C; idx += 256) {
        const int ch = idx % (K / 4) * 4, t = idx / (K / 4), sub = t / SUB;
        float4 k = *reinterpret_cast<const float4*>(gs + t * ROW + ch);
        for (int m = sub + 1; m < NSUB; ++m) {
            const float4 d = *reinterpret_cast<const float4*>(subp + m * K + ch);
            k.x *= d.x; k.y *= d.y; k.z *= d.z; k.w *= d.w;
        }
        *reinterpret_cast<float4*>(gs + t * ROW + ch) = k;
    }
    for (int idx = tid; idx < V / 4 * C; idx += 256) {
        const int col = idx % (V / 4) * 4, t = idx / (V / 4);
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        if (t < rows) load_run<4>(qkv + (size_t)(row0 + t) * p.ld + v_off + col, v);
        const float f = mode == DECAY_STEP ? betas[t] : 1.f;
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = plain ? silu_f(v[e]) : v[e] * f;
        store_run<4>(us + t * V + col, v);
        store_run<4>(ub + t * V + col, v);
    }
    __syncthreads();
    constexpr int RK = K / 64, RV = V / 64;                 // groups of four rows and columns a thread takes
    const int ty = tid >> 4, tx = tid & 15;
    float acc[RK * 4][RV * 4];
#pragma unroll
    for (int i = 0; i < RK * 4; ++i)
#pragma unroll
        for (int j = 0; j < RV * 4; ++j) acc[i][j] = 0.f;
#pragma unroll 2
    for (int t = 0; t < C; ++t) {
        float x[RK * 4], y[RV * 4];
#pragma unroll
        for (int i = 0; i < RK; ++i) {
            const float4 v = *reinterpret_cast<const float4*>(gs + t * ROW + i * 64 + ty * 4);
            x[4 * i] = v.x; x[4 * i + 1] = v.y; x[4 * i + 2] = v.z; x[4 * i + 3] = v.w;
        }
#pragma unroll
        for (int i = 0; i < RV; ++i) {
            const float4 v = *reinterpret_cast<const float4*>(us + t * V + i * 64 + tx * 4);
            y[4 * i] = v.x; y[4 * i + 1] = v.y; y[4 * i + 2] = v.z; y[4 * i + 3] = v.w;
        }
#pragma unroll
        for (int i = 0; i < RK * 4; ++i)
#pragma unroll
            for (int j = 0; j < RV * 4; ++j) acc[i][j] = fmaf(x[i], y[j], acc[i][j]);
    }
    float* dS = p.s + unit * K * V;
#pragma unroll
    for (int i = 0; i < RK * 4; ++i)
#pragma unroll
        for (int j = 0; j < RV; ++j)
            *reinterpret_cast<float4*>(dS + (size_t)((i / 4) * 64 + ty * 4 + i % 4) * V + j * 64 + tx * 4) =
                make_float4(acc[i][4 * j], acc[i][4 * j + 1], acc[i][4 * j + 2], acc[i][4 * j + 3]);
}

// s[chunk] holds what the chunk adds to the state and gets the state in front of the chunk.  A thread four elements,
// grid (K * V / 1024, H, segments).
template <int K, int V>
__global__ void __launch_bounds__(256) chunk_state_kernel(const ChunkArgs p) {
    pdl_launch_dependents();
    const int head = blockIdx.y;
    int row0, rows;
    const int first = first_chunk(p, blockIdx.z, row0, rows);
    if (rows <= 0) return;
    const int chunks = (rows + C - 1) / C;
    const int at = (blockIdx.x * 256 + threadIdx.x) * 4, k = at / V;
    float* dst = p.state + (size_t)p.row_slot[row0] * p.state_stride + (size_t)head * K * V + at;
    pdl_wait();
    float4 S = *reinterpret_cast<const float4*>(dst);
    constexpr int AHEAD = 8;                                // chunks whose shares are on their way
    float4 add[AHEAD];
    float g[AHEAD];
    auto fetch = [&](int c, int slot) {
        const size_t unit = (size_t)(first + c) * p.H + head;
        add[slot] = *reinterpret_cast<const float4*>(p.s + unit * K * V + at);
        g[slot] = p.decay[unit * K + k];
    };
#pragma unroll
    for (int i = 0; i < AHEAD; ++i)
        if (i < chunks) fetch(i, i);
    for (int c0 = 0; c0 < chunks; c0 += AHEAD) {
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) {
            const int c = c0 + i;
            if (c >= chunks) break;
            *reinterpret_cast<float4*>(p.s + ((size_t)(first + c) * p.H + head) * K * V + at) = S;
            S.x = fmaf(S.x, g[i], add[i].x); S.y = fmaf(S.y, g[i], add[i].y);
            S.z = fmaf(S.z, g[i], add[i].z); S.w = fmaf(S.w, g[i], add[i].w);
            if (c + AHEAD < chunks) fetch(c + AHEAD, i);
        }
    }
    *reinterpret_cast<float4*>(dst) = S;
}

template <int K> struct DeltaSmem {
    static constexpr int ROW = K + 16;                      // a token's row: neighbouring rows lie 16 banks apart
    static constexpr int SROW = DCOLS + 4;
    static constexpr size_t bytes = sizeof(float) * (2 * (size_t)C * ROW + 2 * C * DCOLS + K * SROW + K);
};

// The chain of the delta rule: per chunk U = U0 - W S and S <- diag(decay) S + Kd^T U, 16 columns of one head's state a CTA,
// the state and U in shared memory.  Bound by its own two products (512 multiply-adds a thread each, four and two ways
// split along the sum) and four barriers; the operands of the next product are copied while the current one runs.
template <int K, int V>
__global__ void __launch_bounds__(256) chunk_delta_kernel(const ChunkArgs p) {
    constexpr int ROW = DeltaSmem<K>::ROW, SROW = DeltaSmem<K>::SROW;
    extern __shared__ __align__(16) float smem[];
    float* ws = smem;                                       // [C][ROW]
    float* kds = ws + C * ROW;                              // [C][ROW]
    float* u0s = kds + C * ROW;                             // [C][DCOLS]
    float* us = u0s + C * DCOLS;                            // [C][DCOLS]
    float* S = us + C * DCOLS;                              // [K][SROW]
    float* ds = S + K * SROW;                               // [K]
    pdl_launch_dependents();
    const int col0 = blockIdx.x * DCOLS, head = blockIdx.y;
    int row0, rows;
    const int first = first_chunk(p, blockIdx.z, row0, rows);
    if (rows <= 0) return;
    const int chunks = (rows + C - 1) / C;
    const int tid = threadIdx.x;
    float* state = p.state + (size_t)p.row_slot[row0] * p.state_stride + (size_t)head * K * V + col0;
    pdl_wait();
    auto fetch_w = [&](int c) {
        const size_t unit = (size_t)(first + c) * p.H + head;
        for (int i = tid; i < C * K / 4; i += 256)
            copy16(ws + i / (K / 4) * ROW + i % (K / 4) * 4, p.w + unit * C * K + (size_t)i * 4);
        for (int i = tid; i < C * DCOLS / 4; i += 256)
            copy16(u0s + i * 4, p.u + unit * C * V + (size_t)(i / (DCOLS / 4)) * V + col0 + i % (DCOLS / 4) * 4);
        copy_commit();
    };
    auto fetch_kd = [&](int c) {
        const size_t unit = (size_t)(first + c) * p.H + head;
        for (int i = tid; i < C * K / 4; i += 256)
            copy16(kds + i / (K / 4) * ROW + i % (K / 4) * 4, p.kd + unit * C * K + (size_t)i * 4);
        for (int i = tid; i < K / 4; i += 256) copy16(ds + i * 4, p.decay + unit * K + (size_t)i * 4);
        copy_commit();
    };
    fetch_w(0);
    fetch_kd(0);
    for (int i = tid; i < K * DCOLS / 4; i += 256)
        *reinterpret_cast<float4*>(S + i / 4 * SROW + i % 4 * 4) =
            *reinterpret_cast<const float4*>(state + (size_t)(i / 4) * V + i % 4 * 4);
    for (int c = 0; c < chunks; ++c) {
        const size_t unit = (size_t)(first + c) * p.H + head;
        copy_wait<1>();
        __syncthreads();                                    // W, U0 and the state of this chunk are there
        for (int i = tid; i < K * DCOLS / 4; i += 256)
            *reinterpret_cast<float4*>(p.s + unit * K * V + (size_t)(i / 4) * V + col0 + i % 4 * 4) =
                *reinterpret_cast<const float4*>(S + i / 4 * SROW + i % 4 * 4);
        {   // U = U0 - W S: rows rg + 16 i, columns 4 cg.., a quarter of the sum each
            const int cg = tid & 3, kq = (tid >> 2) & 3, rg = tid >> 4;
            float acc[4][4] = {};
#pragma unroll 2
            for (int k0 = 0; k0 < K; k0 += 16) {
                const int k = k0 + kq * 4;
                float4 w[4], s[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) w[i] = *reinterpret_cast<const float4*>(ws + (rg + 16 * i) * ROW + k);
#pragma unroll
                for (int j = 0; j < 4; ++j) s[j] = *reinterpret_cast<const float4*>(S + (k + j) * SROW + cg * 4);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float wi[4] = {w[i].x, w[i].y, w[i].z, w[i].w};
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        acc[i][0] = fmaf(wi[j], s[j].x, acc[i][0]);
                        acc[i][1] = fmaf(wi[j], s[j].y, acc[i][1]);
                        acc[i][2] = fmaf(wi[j], s[j].z, acc[i][2]);
                        acc[i][3] = fmaf(wi[j], s[j].w, acc[i][3]);
                    }
                }
            }
            // the four quarters: every lane ends with one row of its four
            float half[2][4], mine[4];
            const bool up1 = (kq & 1) != 0, up2 = (kq & 2) != 0;
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float give = up1 ? acc[i][e] : acc[i + 2][e], keep = up1 ? acc[i + 2][e] : acc[i][e];
                    half[i][e] = keep + __shfl_xor_sync(0xffffffffu, give, 4);
                }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float give = up2 ? half[0][e] : half[1][e], keep = up2 ? half[1][e] : half[0][e];
                mine[e] = keep + __shfl_xor_sync(0xffffffffu, give, 8);
            }
            const int row = rg + 16 * ((up1 ? 2 : 0) + (up2 ? 1 : 0));
            const float4 u0 = *reinterpret_cast<const float4*>(u0s + row * DCOLS + cg * 4);
            const float4 u = make_float4(u0.x - mine[0], u0.y - mine[1], u0.z - mine[2], u0.w - mine[3]);
            *reinterpret_cast<float4*>(us + row * DCOLS + cg * 4) = u;
            *reinterpret_cast<float4*>(p.u + unit * C * V + (size_t)row * V + col0 + cg * 4) = u;
        }
        __syncthreads();                                    // U is complete, W and U0 are free
        if (c + 1 < chunks) fetch_w(c + 1); else copy_commit();
        copy_wait<1>();
        __syncthreads();                                    // Kd and the decay are there
        {   // S <- diag(decay) S + Kd^T U: rows 4 kg.., columns 4 cg.., every SPLIT-th token
            constexpr int SPLIT = 256 / K;                  // 2 (K 128), 4 (K 64)
            const int cg = tid & 3, sq = (tid >> 2) & (SPLIT - 1), kg = tid / (4 * SPLIT);
            float acc[4][4] = {};
#pragma unroll 4
            for (int t = sq; t < C; t += SPLIT) {
                const float4 kv = *reinterpret_cast<const float4*>(kds + t * ROW + kg * 4);
                const float4 uv = *reinterpret_cast<const float4*>(us + t * DCOLS + cg * 4);
                const float ki[4] = {kv.x, kv.y, kv.z, kv.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    acc[i][0] = fmaf(ki[i], uv.x, acc[i][0]);
                    acc[i][1] = fmaf(ki[i], uv.y, acc[i][1]);
                    acc[i][2] = fmaf(ki[i], uv.z, acc[i][2]);
                    acc[i][3] = fmaf(ki[i], uv.w, acc[i][3]);
                }
            }
            const bool up1 = (sq & 1) != 0, up2 = (sq & 2) != 0;
            float half[2][4];
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float give = up1 ? acc[i][e] : acc[i + 2][e], keep = up1 ? acc[i + 2][e] : acc[i][e];
                    half[i][e] = keep + __shfl_xor_sync(0xffffffffu, give, 4);
                }
            auto add = [&](int k, const float (&v)[4]) {
                float4* at = reinterpret_cast<float4*>(S + k * SROW + cg * 4);
                const float g = ds[k];
                const float4 s = *at;
                *at = make_float4(fmaf(s.x, g, v[0]), fmaf(s.y, g, v[1]), fmaf(s.z, g, v[2]), fmaf(s.w, g, v[3]));
            };
            if (SPLIT == 2) {
                add(kg * 4 + (up1 ? 2 : 0), half[0]);
                add(kg * 4 + (up1 ? 3 : 1), half[1]);
            } else {
                float mine[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float give = up2 ? half[0][e] : half[1][e], keep = up2 ? half[1][e] : half[0][e];
                    mine[e] = keep + __shfl_xor_sync(0xffffffffu, give, 8);
                }
                add(kg * 4 + (up1 ? 2 : 0) + (up2 ? 1 : 0), mine);
            }
        }
        __syncthreads();                                    // the new state is complete, Kd is free
        if (c + 1 < chunks) fetch_kd(c + 1); else copy_commit();
    }
    copy_wait<0>();
    for (int i = tid; i < K * DCOLS / 4; i += 256)
        *reinterpret_cast<float4*>(state + (size_t)(i / 4) * V + i % 4 * 4) =
            *reinterpret_cast<const float4*>(S + i / 4 * SROW + i % 4 * 4);
}

constexpr int OUT_TILE = 32;                    // of the sum, a stage of chunk_output_kernel
constexpr size_t output_smem(int V) { return sizeof(float) * 2 * (size_t)(C * (OUT_TILE + 4) + OUT_TILE * V); }

// o = [q P | A] [S_0; U] of a chunk and head: a warp eight tokens with all value columns, so that a token's norm is a sum
// over its warp; tiles of 32 along the sum, two in flight.  A's part ends at the warp's own tokens.  Modes whose norm is
// not per head leave 32-bit outputs in o_raw.
template <typename T, int K, int V>
__global__ void __launch_bounds__(256) chunk_output_kernel(const ChunkArgs p) {
    constexpr int KT = OUT_TILE, XROW = KT + 4, VC = V / 32;
    extern __shared__ __align__(16) float smem[];
    float* xs = smem;                                       // [2][C][XROW]
    float* ys = smem + 2 * C * XROW;                        // [2][KT][V]
    pdl_launch_dependents();
    const int head = blockIdx.x, chunk = blockIdx.y;
    int row0, rows;
    if (!find_chunk(p, chunk, row0, rows)) return;
    const int tid = threadIdx.x, lane = tid & 31, r0 = (tid >> 5) * 8;
    const size_t unit = (size_t)chunk * p.H + head;
    constexpr int TILES = (K + C) / KT;
    pdl_wait();
    auto fetch = [&](int tile) {
        const int buf = tile & 1, at = tile * KT;
        const float* x = at < K ? p.qb + unit * C * K + at : p.a + unit * C * C + at - K;
        const float* y = at < K ? p.s + unit * K * V + (size_t)at * V : p.u + unit * C * V + (size_t)(at - K) * V;
        const int ldx = at < K ? K : C;
        for (int i = tid; i < C * KT / 4; i += 256)
            copy16(xs + buf * C * XROW + i / (KT / 4) * XROW + i % (KT / 4) * 4, x + (size_t)(i / (KT / 4)) * ldx + i % (KT / 4) * 4);
        for (int i = tid; i < KT * V / 4; i += 256) copy16(ys + buf * KT * V + i * 4, y + (size_t)i * 4);
        copy_commit();
    };
    float acc[8][VC];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int e = 0; e < VC; ++e) acc[i][e] = 0.f;
    fetch(0);
    for (int tile = 0; tile < TILES; ++tile) {
        if (tile + 1 < TILES) fetch(tile + 1); else copy_commit();
        copy_wait<1>();
        __syncthreads();
        const float* x = xs + (tile & 1) * C * XROW;
        const float* y = ys + (tile & 1) * KT * V;
        const int s0 = tile * KT - K;                       // first token of A's columns in this tile (negative: q P)
        const int whole = s0 < 0 ? KT : min(KT, max(0, r0 - s0));           // columns that every token of the warp sees
#pragma unroll 2
        for (int j = 0; j < whole; j += 4) {
            float4 xv[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) xv[i] = *reinterpret_cast<const float4*>(x + (r0 + i) * XROW + j);
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                float yv[VC];
                load_run<VC>(y + (j + m) * V + lane * VC, yv);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float xi = m == 0 ? xv[i].x : m == 1 ? xv[i].y : m == 2 ? xv[i].z : xv[i].w;
#pragma unroll
                    for (int e = 0; e < VC; ++e) acc[i][e] = fmaf(xi, yv[e], acc[i][e]);
                }
            }
        }
        if (s0 >= 0 && r0 >= s0 && r0 < s0 + KT) {          // the warp's own tokens: each sees those up to itself
#pragma unroll
            for (int m = 0; m < 8; ++m) {
                float yv[VC];
                load_run<VC>(y + (r0 - s0 + m) * V + lane * VC, yv);
#pragma unroll
                for (int i = m; i < 8; ++i) {
                    const float xi = x[(r0 + i) * XROW + r0 - s0 + m];
#pragma unroll
                    for (int e = 0; e < VC; ++e) acc[i][e] = fmaf(xi, yv[e], acc[i][e]);
                }
            }
        }
        __syncthreads();
    }
    copy_wait<0>();
    const bool raw = p.mode == DECAY_CONSTANT || p.mode == DECAY_STEP;
    const float* nw = p.norm_w + (p.mode == DECAY_BONUS ? (size_t)head * V : 0) + lane * VC;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        if (r0 + i >= rows) break;
        const size_t rr = (size_t)(row0 + r0 + i);
        if (raw) {
            store_run<VC>(p.o_raw + rr * p.H * V + (size_t)head * V + lane * VC, acc[i]);
            continue;
        }
        float ss = 0.f;
#pragma unroll
        for (int e = 0; e < VC; ++e) ss = fmaf(acc[i][e], acc[i][e], ss);
        ss = warp_sum(ss);
        const float f = rsqrtf(ss / (float)V + p.eps);
        float o[VC], g[VC];
        if (p.gate != nullptr) load_run<VC>((const T*)p.gate + rr * p.ldg + (size_t)head * V + lane * VC, g);
#pragma unroll
        for (int e = 0; e < VC; ++e) {
            o[e] = acc[i][e] * f * nw[e];
            if (p.gate != nullptr) o[e] *= gate_f(g[e], p.gate_act);
        }
        store_run<VC>((T*)p.out + rr * p.ldo + (size_t)head * V + lane * VC, o);
    }
}

template <typename T, int K, int V>
int launch_chunked(const ChunkArgs& p, cudaStream_t stream) {
    const bool delta = p.mode == DECAY_PER_CHANNEL || p.mode == DECAY_PER_HEAD;
    const dim3 per_chunk(p.H, p.chunks);
    const size_t smem = PrepareSmem<K>::bytes(delta);
    if (delta) {
        cudaFuncSetAttribute(chunk_prepare_kernel<T, K, V, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        tis_launch(chunk_prepare_kernel<T, K, V, true>, per_chunk, dim3(256), smem, stream, p);
    } else {
        cudaFuncSetAttribute(chunk_prepare_kernel<T, K, V, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        tis_launch(chunk_prepare_kernel<T, K, V, false>, per_chunk, dim3(256), smem, stream, p);
    }
    int st = tis_check_launch("chunk_prepare");
    if (st != TIS_OK) return st;
    if (delta) {
        cudaFuncSetAttribute(chunk_delta_kernel<K, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DeltaSmem<K>::bytes);
        tis_launch(chunk_delta_kernel<K, V>, dim3(V / DCOLS, p.H, p.segments), dim3(256), DeltaSmem<K>::bytes, stream, p);
    } else {
        tis_launch(chunk_state_kernel<K, V>, dim3(K * V / 1024, p.H, p.segments), dim3(256), 0, stream, p);
    }
    st = tis_check_launch("chunk_state");
    if (st != TIS_OK) return st;
    cudaFuncSetAttribute(chunk_output_kernel<T, K, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)output_smem(V));
    tis_launch(chunk_output_kernel<T, K, V>, per_chunk, dim3(256), output_smem(V), stream, p);
    return tis_check_launch("chunk_output");
}

}  // namespace

// Floats of scratch for a step of n rows in `segments` requests; 0: the chunked kernels do not take these widths.
TIS_API size_t tis_chunked_recurrence_floats(int n, int segments, int H, int k_dim, int v_dim, int delta) {
    if (!((k_dim == 64 || k_dim == 128) && (v_dim == 64 || v_dim == 128)) || n <= 0 || segments <= 0 || H <= 0) return 0;
    const size_t units = ((size_t)n / C + segments) * H;
    return units * ((size_t)C * k_dim * (delta ? 3 : 1) + (size_t)C * v_dim + (size_t)C * C + (size_t)k_dim * v_dim + k_dim);
}

bool chunked_recurrence_takes(int dtype, const ChunkArgs& p, int k_dim, int v_dim) {
    const bool head_step = p.mode == DECAY_PER_HEAD || p.mode == DECAY_STEP || p.mode == DECAY_CONSTANT;
    const bool raw = p.mode == DECAY_CONSTANT || p.mode == DECAY_STEP;
    uintptr_t bases = (uintptr_t)p.qkv | (uintptr_t)p.state;
    if (!head_step) bases |= (uintptr_t)p.a_in;
    if (!raw) bases |= (uintptr_t)p.gate | (uintptr_t)p.out;
    else bases |= (uintptr_t)p.o_raw;
    const bool chunks_fit = p.seg_row0 != nullptr && p.segments > 0 && p.segments <= 65535 && p.H > 0 && p.H <= 65535 && p.G > 0 &&
                            p.H % p.G == 0 && p.n / C + p.segments <= 65535;
    return chunks_fit && (k_dim == 64 || k_dim == 128) && (v_dim == 64 || v_dim == 128) && (dtype == TIS_F32 || dtype == TIS_BF16) &&
           bases % 16 == 0 && p.ld % 8 == 0 && (head_step || p.lda % 8 == 0) && p.state_stride % 4 == 0 &&
           (raw || (p.ldo % 8 == 0 && (p.gate == nullptr || p.ldg % 8 == 0)));
}

int chunked_recurrence(int dtype, ChunkArgs p, int k_dim, int v_dim, float* scratch, size_t scratch_floats, cudaStream_t stream) {
    const bool delta = p.mode == DECAY_PER_CHANNEL || p.mode == DECAY_PER_HEAD;
    p.chunks = p.n / C + p.segments;
    if (scratch == nullptr || (uintptr_t)scratch % 16 != 0 ||
        scratch_floats < tis_chunked_recurrence_floats(p.n, p.segments, p.H, k_dim, v_dim, delta)) {
        tis_set_error("chunked recurrence: %zu floats of scratch for %d rows of %d requests, %d heads", scratch_floats, p.n,
                      p.segments, p.H);
        return TIS_BAD_SIZE;
    }
    const size_t units = (size_t)p.chunks * p.H;
    float* at = scratch;
    auto take = [&](size_t floats) { float* r = at; at += units * floats; return r; };
    p.s = take((size_t)k_dim * v_dim);
    p.qb = take((size_t)C * k_dim);
    p.u = take((size_t)C * v_dim);
    p.a = take((size_t)C * C);
    p.decay = take((size_t)k_dim);
    p.w = delta ? take((size_t)C * k_dim) : nullptr;
    p.kd = delta ? take((size_t)C * k_dim) : nullptr;
#define TIS_CHUNKED(K, V) \
    if (k_dim == K && v_dim == V) TIS_DISPATCH_DTYPE(dtype, T, return (launch_chunked<T, K, V>(p, stream)));
    TIS_CHUNKED(64, 64)
    TIS_CHUNKED(64, 128)
    TIS_CHUNKED(128, 64)
    TIS_CHUNKED(128, 128)
#undef TIS_CHUNKED
    tis_set_error("chunked recurrence: key width %d, value width %d", k_dim, v_dim);
    return TIS_BAD_SIZE;
}
