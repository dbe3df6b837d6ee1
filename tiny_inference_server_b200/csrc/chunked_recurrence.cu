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
// underflows are what they are in the walk.
//
// Numbers that are not finite take other ways through these products than through the walk (a masked zero times an infinity;
// an infinity split in three).  Every one of them, and every sum that overflows on the way, leaves something that is not
// finite in the outputs of its chunk or in the state behind the portion: those two places are looked at, and the walk
// (delta_rule_kernel in seqmix.cu) takes the marked heads of a portion again from the state they began with, which is
// still in the scratch as the state in front of the first chunk.
// Operands, states and sums are 32-bit, with 32-bit and with bfloat16 activations alike: the state goes on from step to step
// whatever the activations are.  The dense products run on the tensor cores as bfloat16 products of operands split in
// three, whose parts hold all 24 bits (mma_split); products of decays are kept as sums of two numbers until they are used.
// Against the walk in 64 bits (2-norms of the difference over the result, five shapes of 128 to 2048 tokens, both
// activations): states 0.5 to 1.05 times as far off as token by token in 32 bits, 32-bit outputs 0.87 to 1.0 times.
// Three tf32 products of operands split in two (2^-22 left out) cost the same tensor time and were 1.1 to 1.7 times as far
// off, with sums left to the tensor cores, which truncate, up to 6.5 times.  On the CUDA cores, which read a word from
// shared memory for every one to four multiply-adds, the kernels took longer (delta rule, 2048 tokens, 12 heads of 128 x 128,
// a layer: 422 us; 271 in tf32, 311 now).
// Straight-line code is kept short: a kernel's code is read anew at every launch, and unrolled over a chunk's tokens the
// exponentials of the preparation took longer to fetch than to run.
#include "recurrence.cuh"

namespace {

constexpr int C = REC_CHUNK, SUB = 16, NSUB = C / SUB;

__device__ __forceinline__ void copy16(void* smem, const void* gmem) {
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

// ---- products of 16 x 16 (x 8) tiles of 32-bit operands in six bfloat16 products.  An operand is the sum of three bfloat16
// numbers (8 + 8 + 8 bits: all of its 24), x = h + m + l; what is left out of a product (m l, l m, l l) is below 2^-26 of it.
// Lane = 4 r + c holds rows r, r + 8 of A (16 x 16) in four columns, column r of B (16 x 8) in the same four, and columns 2 c,
// 2 c + 1 of rows r, r + 8 of the sum.  Which four of the sixteen summed indices is free as long as A and B agree.
// The tensor cores truncate what they add up.  So the sums of every step are added outside, and the large product runs a
// second time with its own rounded sum to be taken off: what the rounding lost, to which the small products are added.
// (A step's sum against 64 bits: 4.8e-8 of its norm with a bias of -3.9e-8 in one chain, 0.7e-8 without a bias so.)
__device__ __forceinline__ void split_pair(float x, float y, unsigned& h, unsigned& m, unsigned& l) {
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(h) : "f"(y), "f"(x));
    x -= __uint_as_float(h << 16); y -= __uint_as_float(h & 0xffff0000u);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(m) : "f"(y), "f"(x));
    x -= __uint_as_float(m << 16); y -= __uint_as_float(m & 0xffff0000u);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(l) : "f"(y), "f"(x));
}
struct FragA {
    unsigned h[4], m[4], l[4];
    // (row r, row r + 8) of the lane's first index, then of its second, third and fourth
    __device__ __forceinline__ void set(float a0, float b0, float a1, float b1, float a2, float b2, float a3, float b3) {
        split_pair(a0, a1, h[0], m[0], l[0]); split_pair(b0, b1, h[1], m[1], l[1]);
        split_pair(a2, a3, h[2], m[2], l[2]); split_pair(b2, b3, h[3], m[3], l[3]);
    }
};
struct FragB {
    unsigned h[2], m[2], l[2];
    __device__ __forceinline__ void set(float b0, float b1, float b2, float b3) {
        split_pair(b0, b1, h[0], m[0], l[0]); split_pair(b2, b3, h[1], m[1], l[1]);
    }
};
__device__ __forceinline__ void mma_bf16(float (&c)[4], const unsigned (&a)[4], const unsigned (&b)[2]) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// c[i] += A B_i for N tiles side by side, up to four at a time; operands(i, b) makes B_i.
template <int N, typename Operands>
__device__ __forceinline__ void mma_split(float (&c)[N][4], const FragA& a, Operands operands) {
    constexpr int G = N < 4 ? N : 4;
#pragma unroll
    for (int i0 = 0; i0 < N; i0 += G) {
        FragB b[G];
        float h[G][4] = {}, d[G][4];
#pragma unroll
        for (int i = 0; i < G; ++i) operands(i0 + i, b[i]);
#pragma unroll
        for (int i = 0; i < G; ++i) mma_bf16(h[i], a.h, b[i].h);
#pragma unroll
        for (int i = 0; i < G; ++i) {
#pragma unroll
            for (int k = 0; k < 4; ++k) d[i][k] = -h[i][k];
            mma_bf16(d[i], a.h, b[i].h);
        }
#pragma unroll
        for (int i = 0; i < G; ++i) mma_bf16(d[i], a.l, b[i].h);
#pragma unroll
        for (int i = 0; i < G; ++i) mma_bf16(d[i], a.h, b[i].l);
#pragma unroll
        for (int i = 0; i < G; ++i) mma_bf16(d[i], a.m, b[i].m);
#pragma unroll
        for (int i = 0; i < G; ++i) mma_bf16(d[i], a.m, b[i].h);
#pragma unroll
        for (int i = 0; i < G; ++i) mma_bf16(d[i], a.h, b[i].m);
#pragma unroll
        for (int i = 0; i < G; ++i)
#pragma unroll
            for (int k = 0; k < 4; ++k) c[i0 + i][k] = (c[i0 + i][k] + d[i][k]) + h[i][k];
    }
}
__device__ __forceinline__ bool finite_f(float x) { return fabsf(x) <= 3.402823466e38f; }

// The rows of segment `seg`, 0 if it is padding or goes on where the one before it ended.
__device__ __forceinline__ int segment_rows(const ChunkArgs& p, int seg, int& row0) {
    row0 = p.seg_row0[seg];
    const int slot = p.row_slot[row0];
    if (slot < 0 || (row0 > 0 && p.row_slot[row0 - 1] == slot)) return 0;
    return p.row_last[row0] - row0 + 1;
}
// Where chunk `chunk` of the step lies (all lanes of a warp together): its first row and number of rows, its segment and that
// segment's first chunk; false: there is no such chunk (the grid is sized by an upper bound).
struct Chunk { int row0, rows, segment, first; };
__device__ __forceinline__ bool find_chunk(const ChunkArgs& p, int chunk, Chunk& at_chunk) {
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
            at_chunk.row0 = __shfl_sync(0xffffffffu, first, at) + in_segment * C;
            at_chunk.rows = min(C, __shfl_sync(0xffffffffu, count, at) - in_segment * C);
            at_chunk.segment = s0 + at;
            at_chunk.first = chunk - in_segment;
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

__host__ __device__ constexpr int m_row(int a) { return SUB * (a + 1) + 4; }    // a row of sub-chunk a's part of M
__host__ __device__ constexpr int m_at(int a) { return 128 * a * (a + 1) + 64 * a; }                // where that part begins
constexpr size_t prepare_smem(int K, bool delta) {
    return sizeof(float) * (3 * (size_t)C * (K + 4) + NSUB * K + 2 * C + 4 + (delta ? m_at(NSUB) : 0));
}

// Two CTAs an SM (shared memory).  Blocks of A and L on the diagonal (16 x 16 tokens) are walked with a running key,
// P(s, t] k_s, four tokens s and a sixteenth of the channels a thread, so that they need neither divisions nor
// exponentials; the others factor at the sub-chunk edges and are products.
template <typename T, int K, int V, bool DELTA>
__global__ void __launch_bounds__(256, 2) chunk_prepare_kernel(const ChunkArgs p) {
    constexpr int ROW = K + 4, CPL = K / 32;                // padding: neighbouring tokens lie four banks apart
    extern __shared__ __align__(16) float smem[];
    float* qs = smem;                                       // [C][ROW]  q, then q P(start of its sub-chunk, t]
    float* ks = qs + C * ROW;                               // k, then the same product
    float* gs = ks + C * ROW;                               // decays, then k P(t, end of its sub-chunk]
    float* subp = gs + C * ROW;                             // [NSUB][K] decay of a whole sub-chunk
    float* betas = subp + NSUB * K;                         // [C]
    float* powers = betas + C;                              // [C + 4] of a constant decay
    float* M = powers + C + 4;                              // diag(beta) L below the diagonal, sub-chunk by sub-chunk
    pdl_launch_dependents();
    const int head = blockIdx.x, chunk = blockIdx.y;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, fr = lane >> 2, fc = lane & 3;
    Chunk here;
    const bool there = find_chunk(p, chunk, here);
    if (chunk == 0) {                                       // nothing is to be taken again so far; who takes which rows
        pdl_wait();
        for (int seg = tid; seg < p.all_segments; seg += 256) {
            const int r = p.seg_row0[seg];
            if (seg < p.segments) p.again[seg * p.H + head] = 0;
            if (p.row_slot[r] >= 0) p.chunked[(size_t)p.row_last[r] * p.H + head] = seg < p.segments;
        }
    }
    if (!there) return;
    const int row0 = here.row0, rows = here.rows;
    const int kvh = head / (p.H / p.G), mode = p.mode;
    const bool forget = mode == DECAY_FORGET_GATE, plain = mode == DECAY_CONSTANT, bonus = mode == DECAY_BONUS;
    const bool per_head = mode == DECAY_PER_HEAD || mode == DECAY_STEP;
    const T* qkv = (const T*)p.qkv;
    const T* a_in = (const T*)p.a_in;
    const int q_off = kvh * K, k_off = p.G * K + kvh * K, v_off = (forget ? 1 : 2) * p.G * K + head * V;
    const float rate = (plain || mode == DECAY_LOG_SIGMOID) ? p.A_log[head] : ((forget || bonus) ? 0.f : expf(p.A_log[head]));
    const int ch0 = lane * CPL;
    if (plain && tid <= C) {                                // each rounded once: an error here is every channel's and every token's
        double power = 1., base = rate;
        for (int e = tid; e > 0; e >>= 1, base *= base)
            if (e & 1) power *= base;
        powers[tid] = (float)power;
    }
    float bias[CPL], low[CPL];
#pragma unroll
    for (int i = 0; i < CPL; ++i) {
        bias[i] = plain ? 0.f : p.dt_bias[per_head ? head : head * K + ch0 + i];
        low[i] = (forget || bonus) ? p.A_log[head * K + ch0 + i] : 0.f;
    }
    pdl_wait();
    // ---- the chunk's token vectors, a warp a token.  First as they are, every load of a thread on its way at once; then
    // token by token in a loop that is short enough to stay in the instruction cache (a token takes some hundred
    // instructions).  A thread reads back what it wrote itself.
#pragma unroll
    for (int u = 0; u < C / 8; ++u) {
        const int t = warp + 8 * u;
        const size_t rr = (size_t)(row0 + min(t, rows - 1));
        float q[CPL], k[CPL], g[CPL];
        load_run<CPL>(qkv + rr * p.ld + q_off + ch0, q);
        load_run<CPL>(forget ? qkv + rr * p.ld + q_off + ch0 : qkv + rr * p.ld + k_off + ch0, k);
        if (!per_head && !plain) load_run<CPL>(a_in + rr * p.lda + (size_t)head * K + ch0, g);
        store_run<CPL>(qs + t * ROW + ch0, q);
        store_run<CPL>(ks + t * ROW + ch0, k);
        if (!per_head && !plain) store_run<CPL>(gs + t * ROW + ch0, g);
    }
    float head_in[2] = {0.f, 0.f};                          // a lane a token: its decay's and its beta's projections
    if (lane < C / 8) {
        const size_t rr = (size_t)(row0 + min(warp + 8 * lane, rows - 1));
        if (per_head) head_in[0] = to_f32(a_in[rr * p.lda + head]);
        if (DELTA) head_in[1] = to_f32(((const T*)p.b_in)[rr * p.ldb + head]);
    }
#pragma unroll 1
    for (int u = 0; u < C / 8; ++u) {
        const int t = warp + 8 * u;
        float q[CPL], k[CPL], g[CPL], beta = 1.f;
        load_run<CPL>(qs + t * ROW + ch0, q);
        load_run<CPL>(ks + t * ROW + ch0, k);
        const float step_in = __shfl_sync(0xffffffffu, head_in[0], u), beta_in = __shfl_sync(0xffffffffu, head_in[1], u);
        if (!per_head && !plain) load_run<CPL>(gs + t * ROW + ch0, g);
        if (DELTA) {
            float sq = 0.f, sk = 0.f;
#pragma unroll
            for (int i = 0; i < CPL; ++i) { sq = fmaf(q[i], q[i], sq); sk = fmaf(k[i], k[i], sk); }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                sq += __shfl_xor_sync(0xffffffffu, sq, o);
                sk += __shfl_xor_sync(0xffffffffu, sk, o);
            }
            const float fq = p.q_scale / sqrtf(sq + p.unit_eps), fk = 1.f / sqrtf(sk + p.unit_eps);
            beta = 1.f / (1.f + expf(-beta_in));
            const float whole = per_head ? expf(-rate * softplus_f(step_in + bias[0])) : 0.f;
#pragma unroll
            for (int i = 0; i < CPL; ++i) {
                g[i] = per_head ? whole : expf(-rate * softplus_f(g[i] + bias[i]));
                q[i] *= fq;
                k[i] *= fk;
            }
        } else if (plain) {
#pragma unroll
            for (int i = 0; i < CPL; ++i) { q[i] = silu_f(q[i]); k[i] = silu_f(k[i]); g[i] = 1.f; }      // (the decays: `powers`)
        } else if (forget) {
#pragma unroll
            for (int i = 0; i < CPL; ++i) {
                const float open = 1.f / (1.f + expf(g[i] + bias[i]));              // 1 - sigmoid of the gate
                q[i] = silu_f(q[i]);
                k[i] = (1.f - low[i]) * open;
                g[i] = low[i] + (1.f - low[i]) * (1.f - open);
            }
        } else if (bonus) {
            float now = 0.f;
#pragma unroll
            for (int i = 0; i < CPL; ++i) {
                q[i] *= p.q_scale;
                g[i] = expf(-expf(g[i] + bias[i]));
                now = fmaf(q[i] * low[i], k[i], now);
            }
            beta = warp_sum(now);
        } else {
            const bool stepped = mode == DECAY_STEP;
            if (stepped) beta = softplus_f(step_in + bias[0]);
            const float whole = stepped ? expf(-rate * beta) : 0.f;
#pragma unroll
            for (int i = 0; i < CPL; ++i) {
                q[i] *= p.q_scale;
                g[i] = stepped ? whole : expf(-rate * softplus_f(-(g[i] + bias[i])));
            }
        }
        if (t >= rows) {                                    // behind the end: changes nothing
#pragma unroll
            for (int i = 0; i < CPL; ++i) { q[i] = 0.f; k[i] = 0.f; g[i] = 1.f; }
            beta = 0.f;
        }
        store_run<CPL>(qs + t * ROW + ch0, q);
        store_run<CPL>(ks + t * ROW + ch0, k);
        store_run<CPL>(gs + t * ROW + ch0, g);
        if (lane == 0) betas[t] = beta;
    }
    __syncthreads();
    const size_t unit = (size_t)chunk * p.H + head;
    float* A = p.a + unit * C * C;
    // ---- blocks on the diagonal: a thread four tokens s.. and every sixteenth float4 of the channels, down the tokens t
    // of its sub-chunk; the sixteen threads of four tokens add their sums up at once
    {
        constexpr int J = K / 64, SUMS = DELTA ? 8 : 4;
        const int slice = tid & 15, grp = tid >> 4, a = grp >> 2, a0 = a * SUB, s0 = a0 + (grp & 3) * 4;
        float4 w[4][J];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < J; ++j) w[i][j] = *reinterpret_cast<const float4*>(ks + (s0 + i) * ROW + j * 64 + slice * 4);
#pragma unroll 2
        for (int t = a0 + (s0 & 8); t < a0 + SUB; ++t) {
            float4 q[J], k[J], g[J];
#pragma unroll
            for (int j = 0; j < J; ++j) {
                const int at = t * ROW + j * 64 + slice * 4;
                q[j] = *reinterpret_cast<const float4*>(qs + at);
                g[j] = *reinterpret_cast<const float4*>(gs + at);
                if (DELTA) k[j] = *reinterpret_cast<const float4*>(ks + at);
            }
            float sum[SUMS];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const bool later = t > s0 + i;
                if (!bonus && later) {
#pragma unroll
                    for (int j = 0; j < J; ++j) { w[i][j].x *= g[j].x; w[i][j].y *= g[j].y; w[i][j].z *= g[j].z; w[i][j].w *= g[j].w; }
                }
                float da = 0.f, db = 0.f, la = 0.f, lb = 0.f;
#pragma unroll
                for (int j = 0; j < J; ++j) {
                    da = fmaf(q[j].x, w[i][j].x, fmaf(q[j].y, w[i][j].y, da));
                    db = fmaf(q[j].z, w[i][j].z, fmaf(q[j].w, w[i][j].w, db));
                    if (DELTA) {
                        la = fmaf(k[j].x, w[i][j].x, fmaf(k[j].y, w[i][j].y, la));
                        lb = fmaf(k[j].z, w[i][j].z, fmaf(k[j].w, w[i][j].w, lb));
                    }
                }
                sum[i] = da + db;
                if (DELTA) sum[SUMS - 4 + i] = la + lb;
                if (bonus && later) {
#pragma unroll
                    for (int j = 0; j < J; ++j) { w[i][j].x *= g[j].x; w[i][j].y *= g[j].y; w[i][j].z *= g[j].z; w[i][j].w *= g[j].w; }
                }
            }
            int which = 0;
#pragma unroll
            for (int half = SUMS / 2, o = 8; o > 0; half >>= 1, o >>= 1) {
                if (half > 0) {
                    const bool upper = (slice & o) != 0;
#pragma unroll
                    for (int i = 0; i < SUMS / 2; ++i)
                        if (i < half) {
                            const float give = upper ? sum[i] : sum[i + half], keep = upper ? sum[i + half] : sum[i];
                            sum[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
                        }
                    which += upper ? half : 0;
                } else {
                    sum[0] += __shfl_xor_sync(0xffffffffu, sum[0], o);
                }
            }
            const int s = s0 + (which & 3);
            if ((slice & (DELTA ? 1 : 3)) == 0) {
                if (which < 4) {
                    if (t >= s) A[t * C + s] = (bonus && t == s) ? betas[t] : (plain ? sum[0] * powers[t - s] : sum[0]);
                } else if (t > s) {
                    M[m_at(a) + (t - a0) * m_row(a) + s] = betas[t] * sum[0];
                }
            }
        }
    }
    __syncthreads();
    // ---- products of decays inside the sub-chunks, as sums of two numbers: each has one rounding in the end, not one a token
    for (int idx = tid; idx < K * NSUB; idx += 256) {
        const int ch = idx % K, sub = idx / K, live = min(SUB, max(0, rows - sub * SUB));
        float g[SUB], k[SUB], hi = 1.f, lo = 0.f;
        auto times = [&](float x) {
            const float p = hi * x;
            lo = fmaf(lo, x, fmaf(hi, x, -p));
            hi = p;
        };
#pragma unroll
        for (int r = 0; r < SUB; ++r) {
            const int at = (sub * SUB + r) * ROW + ch;
            g[r] = gs[at];
            k[r] = ks[at];
            if (plain) hi = powers[min(r + 1, live)];
            else if (!bonus) times(g[r]);
            qs[at] = fmaf(qs[at], hi, qs[at] * lo);
            if (DELTA) ks[at] = fmaf(k[r], hi, k[r] * lo);
            if (bonus) times(g[r]);
        }
        subp[sub * K + ch] = hi + lo;
        hi = 1.f; lo = 0.f;
#pragma unroll
        for (int r = SUB - 1; r >= 0; --r) {
            if (plain) hi = powers[max(0, live - 1 - r)];
            gs[(sub * SUB + r) * ROW + ch] = fmaf(k[r], hi, k[r] * lo);
            if (!plain) times(g[r]);
        }
    }
    __syncthreads();
    // ---- blocks below the diagonal: a warp each
    if (warp < 6) {
        const int a = warp < 3 ? 3 : (warp < 5 ? 2 : 1), b = warp < 3 ? warp : (warp < 5 ? warp - 3 : 0);
        const int t0 = a * SUB + fr, s0 = b * SUB + fr;
        float acc[2][4] = {}, accl[2][4] = {};
        auto rows_of = [&](const float* x, int c, FragA& f) {
            const float *x0 = x + t0 * ROW + c, *x8 = x0 + 8 * ROW;
            f.set(x0[0], x8[0], x0[4], x8[4], x0[8], x8[8], x0[12], x8[12]);
        };
#pragma unroll 2
        for (int c = fc; c < K; c += 16) {
            float f[4];                                     // whole sub-chunks between the two
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                f[e] = 1.f;
                for (int m = b + 1; m < a; ++m) f[e] *= subp[m * K + c + 4 * e];
            }
            FragB kb[2];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const float* k = gs + (s0 + 8 * j) * ROW + c;
                kb[j].set(k[0] * f[0], k[4] * f[1], k[8] * f[2], k[12] * f[3]);
            }
            FragA x;
            rows_of(qs, c, x);
            mma_split<2>(acc, x, [&](int j, FragB& o) { o = kb[j]; });
            if (DELTA) {
                rows_of(ks, c, x);
                mma_split<2>(accl, x, [&](int j, FragB& o) { o = kb[j]; });
            }
        }
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int t = t0 + 8 * i, s = b * SUB + 8 * j + 2 * fc;
                *reinterpret_cast<float2*>(A + t * C + s) = make_float2(acc[j][2 * i], acc[j][2 * i + 1]);
                if (DELTA)
                    *reinterpret_cast<float2*>(M + m_at(a) + (t - a * SUB) * m_row(a) + s) =
                        make_float2(betas[t] * accl[j][2 * i], betas[t] * accl[j][2 * i + 1]);
            }
    } else if (DELTA) {
        // meanwhile: (I + M)^-1 - I of the blocks on the diagonal, in their place, a thread a column
        const int i = tid - 192, a = i >> 4, j = i & 15;
        float* m = M + m_at(a) + a * SUB;
        float x[SUB];
#pragma unroll
        for (int t = 0; t < SUB; ++t) {
            float y = t == j ? 1.f : 0.f;
#pragma unroll
            for (int s = 0; s < t; ++s) y = fmaf(-m[t * m_row(a) + s], x[s], y);
            x[t] = t < j ? 0.f : y;
        }
        __syncwarp();
#pragma unroll
        for (int t = 0; t < SUB; ++t) m[t * m_row(a) + j] = t > j ? x[t] : 0.f;
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
        p.decay[unit * K + ch] = plain ? powers[min(C, rows)] : d;
    }
    float* ub = p.u + unit * C * V;
    __syncthreads();                                        // qs is written out, gs and M are complete
    float* kd = DELTA ? p.kd + unit * C * K : gs;
    for (int idx = tid; idx < K / 4 * C; idx += 256) {
        const int ch = idx % (K / 4) * 4, t = idx / (K / 4), sub = t / SUB;
        float4 k = *reinterpret_cast<const float4*>(gs + t * ROW + ch);
        for (int m = sub + 1; m < NSUB; ++m) {
            const float4 d = *reinterpret_cast<const float4*>(subp + m * K + ch);
            k.x *= d.x; k.y *= d.y; k.z *= d.z; k.w *= d.w;
        }
        *reinterpret_cast<float4*>(kd + t * (DELTA ? K : ROW) + ch) = k;
    }
    if (DELTA) {
        // the triangular system, 16 columns of [beta K P(0, .] | beta V] a warp, transposed: the sums of one block of
        // tokens are, lane by lane, the operands of the next
        for (int tile = warp; tile < (K + V) / 16; tile += 8) {
            const bool key = tile < K / 16;
            const int col = (key ? tile : tile - K / 16) * 16 + fr;
            float x[C / 8][4];
            float pre[2] = {1.f, 1.f};
#pragma unroll
            for (int j = 0; j < C / 8; ++j) {
                if (key && j > 0 && j % 2 == 0) { pre[0] *= subp[(j / 2 - 1) * K + col]; pre[1] *= subp[(j / 2 - 1) * K + col + 8]; }
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int t = 8 * j + 2 * fc + (e & 1), c = col + (e >> 1) * 8;
                    x[j][e] = key ? ks[t * ROW + c] * pre[e >> 1]
                                  : to_f32(qkv[(size_t)(row0 + min(t, rows - 1)) * p.ld + v_off + c]);
                }
            }
#pragma unroll
            for (int j = 0; j < C / 8; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int t = 8 * j + 2 * fc + (e & 1);
                    x[j][e] = t < rows ? x[j][e] * betas[t] : 0.f;
                }
#pragma unroll
            for (int a = 0; a < NSUB; ++a) {
                const float* m = M + m_at(a) + fr * m_row(a) + 2 * fc;
                // (what earlier blocks take away is summed apart: a sum of smaller numbers, rounded finer)
                float y[2][4], less[2][4] = {};
#pragma unroll
                for (int j = 0; j < 2 * a; j += 2) {
                    FragA f;
                    f.set(x[j][0], x[j][2], x[j][1], x[j][3], x[j + 1][0], x[j + 1][2], x[j + 1][1], x[j + 1][3]);
                    mma_split<2>(less, f, [&](int i, FragB& o) {
                        const float2 v = *reinterpret_cast<const float2*>(m + 8 * i * m_row(a) + 8 * j);
                        const float2 w = *reinterpret_cast<const float2*>(m + 8 * i * m_row(a) + 8 * j + 8);
                        o.set(v.x, v.y, w.x, w.y);
                    });
                }
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int e = 0; e < 4; ++e) y[i][e] = x[2 * a + i][e] - less[i][e];
                FragA f;
                f.set(y[0][0], y[0][2], y[0][1], y[0][3], y[1][0], y[1][2], y[1][1], y[1][3]);
                float more[2][4] = {};
                mma_split<2>(more, f, [&](int i, FragB& o) {
                    const float2 v = *reinterpret_cast<const float2*>(m + 8 * i * m_row(a) + a * SUB);
                    const float2 w = *reinterpret_cast<const float2*>(m + 8 * i * m_row(a) + a * SUB + 8);
                    o.set(v.x, v.y, w.x, w.y);
                });
#pragma unroll
                for (int e = 0; e < 4; ++e) { x[2 * a][e] = y[0][e] + more[0][e]; x[2 * a + 1][e] = y[1][e] + more[1][e]; }
            }
            float* dst = key ? p.w + unit * C * K : ub;
            const int ldd = key ? K : V;
#pragma unroll
            for (int j = 0; j < C / 8; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) dst[(8 * j + 2 * fc + (e & 1)) * ldd + col + (e >> 1) * 8] = x[j][e];
        }
        return;
    }
    // ---- the chunk's share of the state, sum_s (k_s P(s, C]) u_s^T
    constexpr int UROW = V + 4;
    float* us = smem;                                       // [C][UROW], over the queries and keys
    for (int idx = tid; idx < V / 4 * C; idx += 256) {
        const int col = idx % (V / 4) * 4, t = idx / (V / 4);
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        if (t < rows) load_run<4>(qkv + (size_t)(row0 + t) * p.ld + v_off + col, v);
        const float f = mode == DECAY_STEP ? betas[t] : 1.f;
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = plain ? silu_f(v[e]) : v[e] * f;
        store_run<4>(us + t * UROW + col, v);
        store_run<4>(ub + t * V + col, v);
    }
    __syncthreads();
    constexpr int MW = K / 32, NT = V / 8 / (8 / MW);       // warps along the channels (32 each), column tiles of a warp
    const int mb = (warp % MW) * 32, nb = (warp / MW) * NT * 8;
    float acc[2][NT][4] = {};
#pragma unroll 1
    for (int t0 = 0; t0 < C; t0 += 16) {
        const int t = t0 + 2 * fc;                          // a lane's tokens: t, t + 1, t + 8, t + 9
        FragA f[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const float *at = gs + t * ROW + mb + 16 * i + fr, *at8 = at + 8 * ROW;
            f[i].set(at[0], at[8], at[ROW], at[ROW + 8], at8[0], at8[8], at8[ROW], at8[ROW + 8]);
        }
#pragma unroll
        for (int j = 0; j < NT; j += 2) {
            FragB u[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const float* at = us + t * UROW + nb + 8 * (j + e) + fr;
                u[e].set(at[0], at[UROW], at[8 * UROW], at[9 * UROW]);
            }
#pragma unroll
            for (int i = 0; i < 2; ++i)
                mma_split<2>(reinterpret_cast<float(&)[2][4]>(acc[i][j]), f[i], [&](int e, FragB& o) { o = u[e]; });
        }
    }
    float* dS = p.s + unit * K * V;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h)
                *reinterpret_cast<float2*>(dS + (size_t)(mb + 16 * i + 8 * h + fr) * V + nb + 8 * j + 2 * fc) =
                    make_float2(acc[i][j][2 * h], acc[i][j][2 * h + 1]);
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
    if (!(finite_f(S.x) && finite_f(S.y) && finite_f(S.z) && finite_f(S.w))) p.again[blockIdx.z * p.H + head] = first + 1;
}

template <int K, int NT> struct DeltaSmem {
    static constexpr int ROW = K + 4, COLS = 8 * NT;
    static constexpr int SROW = COLS + 8, UROW = COLS + 4;  // rows of the state and of U: fragments meet every bank once
    static constexpr int STAGE = 2 * C * ROW + C * COLS + K;                    // W, Kd, U0, decay of a chunk
    static constexpr size_t bytes = sizeof(float) * (2 * (size_t)STAGE + C * UROW + K * SROW);
};

// The chain of the delta rule: per chunk U = U0 - W S and S <- diag(decay) S + Kd^T U, 8 NT columns of one head's state a
// CTA.  The state lives in the registers of the warps that sum it and, for the next chunk's first product, in shared
// memory; the next chunk's operands are copied while this one's run.  Bound by the chain of the two products (seven tensor
// instructions a step of 16 along the sum) and what stands between them: two barriers, the operands' split.
template <int K, int V, int NT>
__global__ void __launch_bounds__(256, 1) chunk_delta_kernel(const ChunkArgs p) {
    typedef DeltaSmem<K, NT> L;
    constexpr int ROW = L::ROW, COLS = L::COLS, SROW = L::SROW, UROW = L::UROW;
    extern __shared__ __align__(16) float smem[];
    float* us = smem + 2 * L::STAGE;                        // [C][UROW]
    float* S = us + C * UROW;                               // [K][SROW]
    pdl_launch_dependents();
    const int col0 = blockIdx.x * COLS, head = blockIdx.y;
    int row0, rows;
    const int first = first_chunk(p, blockIdx.z, row0, rows);
    if (rows <= 0) return;
    const int chunks = (rows + C - 1) / C;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, fr = lane >> 2, fc = lane & 3;
    float* state = p.state + (size_t)p.row_slot[row0] * p.state_stride + (size_t)head * K * V + col0;
    pdl_wait();
    auto fetch = [&](int c) {
        const size_t unit = (size_t)(first + c) * p.H + head;
        float* ws = smem + (c & 1) * L::STAGE;
        float* kds = ws + C * ROW;
        float* u0s = kds + C * ROW;
        float* ds = u0s + C * COLS;
        for (int i = tid; i < C * K / 4; i += 256) copy16(ws + i / (K / 4) * ROW + i % (K / 4) * 4, p.w + unit * C * K + (size_t)i * 4);
        for (int i = tid; i < C * COLS / 4; i += 256)
            copy16(u0s + i * 4, p.u + unit * C * V + (size_t)(i / (COLS / 4)) * V + col0 + i % (COLS / 4) * 4);
        for (int i = tid; i < C * K / 4; i += 256) copy16(kds + i / (K / 4) * ROW + i % (K / 4) * 4, p.kd + unit * C * K + (size_t)i * 4);
        for (int i = tid; i < K / 4; i += 256) copy16(ds + i * 4, p.decay + unit * K + (size_t)i * 4);
        copy_commit();
    };
    fetch(0);
    // the part of the state that this warp sums: rows sm.., SN column tiles from sn on
    constexpr int SM = K / 16, SW = 8 / SM, SN = NT / SW;   // row tiles, warps that share one, column tiles of each
    const int sm = warp / SW * 16, sn = warp % SW * SN * 8;
    float s[SN][4];
#pragma unroll
    for (int j = 0; j < SN; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float2 v = *reinterpret_cast<const float2*>(state + (size_t)(sm + fr + 8 * h) * V + sn + 8 * j + 2 * fc);
            s[j][2 * h] = v.x; s[j][2 * h + 1] = v.y;
        }
    // the part of U that this warp sums: tokens um.., half of the column tiles
    constexpr int UN = NT / 2;
    const int um = (warp & 3) * 16, un = (warp >> 2) * UN * 8;
    for (int c = 0; c < chunks; ++c) {
        const size_t unit = (size_t)(first + c) * p.H + head;
        const float* ws = smem + (c & 1) * L::STAGE;
        const float* kds = ws + C * ROW;
        const float* u0s = kds + C * ROW;
        const float* ds = u0s + C * COLS;
#pragma unroll
        for (int j = 0; j < SN; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float2 v = make_float2(s[j][2 * h], s[j][2 * h + 1]);
                const int k = sm + fr + 8 * h, col = sn + 8 * j + 2 * fc;
                *reinterpret_cast<float2*>(S + k * SROW + col) = v;
                *reinterpret_cast<float2*>(p.s + unit * K * V + (size_t)k * V + col0 + col) = v;
            }
        copy_wait<0>();
        __syncthreads();                                    // the chunk's operands and the state; the other stage is free
        if (c + 1 < chunks) fetch(c + 1);
        {   // U = U0 - W S
            float acc[UN][4] = {};
#pragma unroll
            for (int k0 = 0; k0 < K; k0 += 16) {
                const int k = k0 + fc;
                const float *w = ws + (um + fr) * ROW + k, *w8 = w + 8 * ROW;
                FragA f;
                f.set(w[0], w8[0], w[4], w8[4], w[8], w8[8], w[12], w8[12]);
                mma_split<UN>(acc, f, [&](int j, FragB& o) {
                    const float* at = S + k * SROW + un + 8 * j + fr;
                    o.set(at[0], at[4 * SROW], at[8 * SROW], at[12 * SROW]);
                });
            }
#pragma unroll
            for (int j = 0; j < UN; ++j)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int t = um + fr + 8 * h, col = un + 8 * j + 2 * fc;
                    const float2 u0 = *reinterpret_cast<const float2*>(u0s + t * COLS + col);
                    const float2 u = make_float2(u0.x - acc[j][2 * h], u0.y - acc[j][2 * h + 1]);
                    *reinterpret_cast<float2*>(us + t * UROW + col) = u;
                    *reinterpret_cast<float2*>(p.u + unit * C * V + (size_t)t * V + col0 + col) = u;
                }
        }
        __syncthreads();                                    // U is complete, nobody reads the state any more
        {   // S <- diag(decay) S + Kd^T U
            float acc[SN][4] = {};
#pragma unroll
            for (int t0 = 0; t0 < C; t0 += 16) {
                const int t = t0 + 2 * fc;
                const float *kd = kds + t * ROW + sm + fr, *kd8 = kd + 8 * ROW;
                FragA f;
                f.set(kd[0], kd[8], kd[ROW], kd[ROW + 8], kd8[0], kd8[8], kd8[ROW], kd8[ROW + 8]);
                mma_split<SN>(acc, f, [&](int j, FragB& o) {
                    const float* at = us + t * UROW + sn + 8 * j + fr;
                    o.set(at[0], at[UROW], at[8 * UROW], at[9 * UROW]);
                });
            }
            const float g0 = ds[sm + fr], g1 = ds[sm + fr + 8];
#pragma unroll
            for (int j = 0; j < SN; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) s[j][e] = fmaf(s[j][e], e < 2 ? g0 : g1, acc[j][e]);
        }
    }
    bool fine = true;
#pragma unroll
    for (int j = 0; j < SN; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            *reinterpret_cast<float2*>(state + (size_t)(sm + fr + 8 * h) * V + sn + 8 * j + 2 * fc) =
                make_float2(s[j][2 * h], s[j][2 * h + 1]);
            fine = fine && finite_f(s[j][2 * h]) && finite_f(s[j][2 * h + 1]);
        }
    if (!fine) p.again[blockIdx.z * p.H + head] = first + 1;
}

constexpr int OUT_TILE = 32;                    // of the sum, a stage of chunk_output_kernel
constexpr size_t output_smem(int V, size_t type) {
    return sizeof(float) * 2 * (size_t)(C * (OUT_TILE + 4) + OUT_TILE * (V + 8)) + type * C * V;
}

// o = [q P | A] [S_0; U] of a chunk and head: a warp a sub-chunk's 16 tokens and half of the value columns; tiles of 32 along
// the sum, two in flight.  A's part ends with the warp's own tokens.  Modes whose norm is not per head leave 32-bit
// outputs in o_raw.
template <typename T, int K, int V>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 2 : 3) chunk_output_kernel(const ChunkArgs p) {
    constexpr int KT = OUT_TILE, XROW = KT + 4, YROW = V + 8, NT = V / 16;
    extern __shared__ __align__(16) float smem[];
    float* xs = smem;                                       // [2][C][XROW]
    float* ys = smem + 2 * C * XROW;                        // [2][KT][YROW]
    T* gs = reinterpret_cast<T*>(ys + 2 * KT * YROW);       // [C][V]
    pdl_launch_dependents();
    const int head = blockIdx.x, chunk = blockIdx.y;
    Chunk here;
    if (!find_chunk(p, chunk, here)) return;
    const int row0 = here.row0, rows = here.rows;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, fr = lane >> 2, fc = lane & 3;
    const int a = warp & 3, r0 = a * SUB + fr, n0 = (warp >> 2) * (V / 2);
    const size_t unit = (size_t)chunk * p.H + head;
    constexpr int TILES = (K + C) / KT;
    const bool raw = p.mode == DECAY_CONSTANT || p.mode == DECAY_STEP, gated = !raw && p.gate != nullptr;
    pdl_wait();
    if (gated) {                                            // what the last step reads, on its way from the beginning
        constexpr int PER = 16 / (int)sizeof(T);
        for (int i = tid; i < C * V / PER; i += 256) {
            const int t = i / (V / PER), at = i % (V / PER) * PER;
            copy16(gs + t * V + at, (const T*)p.gate + (size_t)(row0 + min(t, rows - 1)) * p.ldg + (size_t)head * V + at);
        }
    }
    auto fetch = [&](int tile) {
        const int buf = tile & 1, at = tile * KT;
        const float* x = at < K ? p.qb + unit * C * K + at : p.a + unit * C * C + at - K;
        const float* y = at < K ? p.s + unit * K * V + (size_t)at * V : p.u + unit * C * V + (size_t)(at - K) * V;
        const int ldx = at < K ? K : C;
        for (int i = tid; i < C * KT / 4; i += 256)
            copy16(xs + buf * C * XROW + i / (KT / 4) * XROW + i % (KT / 4) * 4, x + (size_t)(i / (KT / 4)) * ldx + i % (KT / 4) * 4);
        for (int i = tid; i < KT * V / 4; i += 256)
            copy16(ys + buf * KT * YROW + i / (V / 4) * YROW + i % (V / 4) * 4, y + (size_t)i * 4);
        copy_commit();
    };
    float acc[NT][4] = {};
    fetch(0);
    for (int tile = 0; tile < TILES; ++tile) {
        if (tile + 1 < TILES) fetch(tile + 1); else copy_commit();
        copy_wait<1>();
        __syncthreads();
        const float* x = xs + (tile & 1) * C * XROW + r0 * XROW;
        const float* y = ys + (tile & 1) * KT * YROW + n0 + fr;
        const int s0 = tile * KT - K;                       // first token of A's columns in this tile (negative: q P)
        const int whole = s0 < 0 ? KT : min(KT, max(0, a * SUB - s0));      // columns that every token of the warp sees
        auto column = [&](int k, int i, FragB& o) {
            const float* at = y + k * YROW + 8 * i;
            o.set(at[0], at[4 * YROW], at[8 * YROW], at[12 * YROW]);
        };
#pragma unroll 1
        for (int j = 0; j < whole; j += 16) {
            const int k = j + fc;
            const float* x8 = x + 8 * XROW;
            FragA f;
            f.set(x[k], x8[k], x[k + 4], x8[k + 4], x[k + 8], x8[k + 8], x[k + 12], x8[k + 12]);
            mma_split<NT>(acc, f, [&](int i, FragB& o) { column(k, i, o); });
        }
        const int d0 = a * SUB - s0;                        // where the warp's own tokens lie in this tile
        if (s0 >= 0 && d0 >= 0 && d0 < KT) {
            const int k = d0 + fc;
            float v[8];                                 // a token sees those up to itself
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                v[2 * e] = fr >= fc + 4 * e ? x[k + 4 * e] : 0.f;
                v[2 * e + 1] = fr + 8 >= fc + 4 * e ? x[8 * XROW + k + 4 * e] : 0.f;
            }
            FragA f;
            f.set(v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7]);
            mma_split<NT>(acc, f, [&](int i, FragB& o) { column(k, i, o); });
        }
        __syncthreads();
    }
    copy_wait<0>();
    // through shared memory, so that a warp has eight whole tokens: their norms, gates and stores
    constexpr int OROW = V + 4, VC = V / 32;
    float* os = smem;                                       // [C][OROW], over the tiles
    bool fine = true;
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) fine = fine && finite_f(acc[i][e]);
    if (!fine) p.again[here.segment * p.H + head] = here.first + 1;
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h)
            *reinterpret_cast<float2*>(os + (r0 + 8 * h) * OROW + n0 + 8 * i + 2 * fc) = make_float2(acc[i][2 * h], acc[i][2 * h + 1]);
    const int t0 = warp * 8, col = lane * VC;
    float nw[VC];
#pragma unroll
    for (int e = 0; e < VC; ++e) nw[e] = raw ? 1.f : p.norm_w[(p.mode == DECAY_BONUS ? head * V : 0) + col + e];
    __syncthreads();
    const int count = min(8, rows - t0);
#pragma unroll 1
    for (int i = 0; i < count; ++i) {                       // (a loop that stays in the instruction cache)
        const size_t rr = (size_t)(row0 + t0 + i);
        float o[VC];
        load_run<VC>(os + (t0 + i) * OROW + col, o);
        if (raw) {
            store_run<VC>(p.o_raw + rr * p.H * V + (size_t)head * V + col, o);
            continue;
        }
        float ss = 0.f;
#pragma unroll
        for (int e = 0; e < VC; ++e) ss = fmaf(o[e], o[e], ss);
        ss = warp_sum(ss);
        const float f = rsqrtf(ss / (float)V + p.eps);
        float g[VC];
        if (gated) load_run<VC>(gs + (t0 + i) * V + col, g);
#pragma unroll
        for (int e = 0; e < VC; ++e) {
            o[e] = o[e] * f * nw[e];
            if (gated) o[e] *= gate_f(g[e], p.gate_act);
        }
        store_run<VC>((T*)p.out + rr * p.ldo + (size_t)head * V + col, o);
    }
}

template <typename T, int K, int V>
int launch_chunked(const ChunkArgs& p, cudaStream_t stream) {
    const bool delta = p.mode == DECAY_PER_CHANNEL || p.mode == DECAY_PER_HEAD;
    const dim3 per_chunk(p.H, p.chunks);
    const size_t smem = prepare_smem(K, delta);
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
        // 16 columns a CTA while all CTAs are resident (one an SM), else 32
        if (p.H * (V / 16) * p.segments <= 148) {
            cudaFuncSetAttribute(chunk_delta_kernel<K, V, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DeltaSmem<K, 2>::bytes);
            tis_launch(chunk_delta_kernel<K, V, 2>, dim3(V / 16, p.H, p.segments), dim3(256), DeltaSmem<K, 2>::bytes, stream, p);
        } else {
            cudaFuncSetAttribute(chunk_delta_kernel<K, V, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DeltaSmem<K, 4>::bytes);
            tis_launch(chunk_delta_kernel<K, V, 4>, dim3(V / 32, p.H, p.segments), dim3(256), DeltaSmem<K, 4>::bytes, stream, p);
        }
    } else {
        tis_launch(chunk_state_kernel<K, V>, dim3(K * V / 1024, p.H, p.segments), dim3(256), 0, stream, p);
    }
    st = tis_check_launch("chunk_state");
    if (st != TIS_OK) return st;
    cudaFuncSetAttribute(chunk_output_kernel<T, K, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)output_smem(V, sizeof(T)));
    tis_launch(chunk_output_kernel<T, K, V>, per_chunk, dim3(256), output_smem(V, sizeof(T)), stream, p);
    return tis_check_launch("chunk_output");
}

}  // namespace

bool chunked_recurrence_takes(int dtype, const ChunkArgs& p, int k_dim, int v_dim) {
    const bool head_step = p.mode == DECAY_PER_HEAD || p.mode == DECAY_STEP || p.mode == DECAY_CONSTANT;
    const bool raw = p.mode == DECAY_CONSTANT || p.mode == DECAY_STEP;
    uintptr_t bases = (uintptr_t)p.qkv | (uintptr_t)p.state;
    if (!head_step) bases |= (uintptr_t)p.a_in;
    if (!raw) bases |= (uintptr_t)p.gate | (uintptr_t)p.out;
    else bases |= (uintptr_t)p.o_raw;
    const bool chunks_fit = p.segments > 0 && p.segments <= 65535 && p.H > 0 && p.H <= 65535 && p.G > 0 &&
                            p.H % p.G == 0 && p.n > 0 && p.n / C + p.segments <= 65535;
    return chunks_fit && (k_dim == 64 || k_dim == 128) && (v_dim == 64 || v_dim == 128) && (dtype == TIS_F32 || dtype == TIS_BF16) &&
           bases % 16 == 0 && p.ld % 8 == 0 && (head_step || p.lda % 8 == 0) && p.state_stride % 4 == 0 &&
           (raw || (p.ldo % 8 == 0 && (p.gate == nullptr || p.ldg % 8 == 0)));
}

// Floats of scratch for p.n rows in p.segments portions of a step of p.all_rows rows, and the arrays in it.
static size_t chunk_arrays(ChunkArgs& p, int k_dim, int v_dim, float* scratch) {
    const bool delta = p.mode == DECAY_PER_CHANNEL || p.mode == DECAY_PER_HEAD;
    p.chunks = p.n / C + p.segments;
    const size_t units = (size_t)p.chunks * p.H;
    size_t at = 0;
    auto take = [&](size_t floats) { float* r = scratch + at; at += (floats + 3) / 4 * 4; return r; };
    p.s = take(units * k_dim * v_dim);
    p.qb = take(units * C * k_dim);
    p.u = take(units * C * v_dim);
    p.a = take(units * C * C);
    p.decay = take(units * k_dim);
    p.w = delta ? take(units * C * k_dim) : nullptr;
    p.kd = delta ? take(units * C * k_dim) : nullptr;
    p.again = reinterpret_cast<int*>(take((size_t)p.segments * p.H));
    p.chunked = reinterpret_cast<int*>(take((size_t)p.all_rows * p.H));
    return at;
}
// Floats of scratch for `rows` rows in `segments` portions of a step of `all_rows` rows; 0: the chunked kernels do not take these
// operands (o_raw lies on a 16-byte boundary).
TIS_API size_t tis_chunked_recurrence_floats(int dtype, int mode, const void* qkv, int ld, const void* a_in, int lda, const void* gate,
                                             int ldg, const void* out, int ldo, const float* state, size_t state_stride, int rows,
                                             int segments, int all_rows, int H, int G, int k_dim, int v_dim) {
    ChunkArgs p = {};
    p.qkv = qkv; p.ld = ld; p.a_in = a_in; p.lda = lda; p.gate = gate; p.ldg = ldg; p.out = const_cast<void*>(out); p.ldo = ldo;
    p.state = const_cast<float*>(state); p.state_stride = state_stride; p.n = rows; p.segments = segments; p.all_rows = all_rows;
    p.H = H; p.G = G; p.mode = mode;
    return chunked_recurrence_takes(dtype, p, k_dim, v_dim) ? chunk_arrays(p, k_dim, v_dim, nullptr) : 0;
}

int chunked_recurrence(int dtype, ChunkArgs& p, int k_dim, int v_dim, float* scratch, size_t scratch_floats, cudaStream_t stream) {
    if (scratch == nullptr || (uintptr_t)scratch % 16 != 0 || scratch_floats < chunk_arrays(p, k_dim, v_dim, scratch)) {
        tis_set_error("chunked recurrence: %zu floats of scratch for %d rows of %d requests, %d heads", scratch_floats, p.n,
                      p.segments, p.H);
        return TIS_BAD_SIZE;
    }
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
