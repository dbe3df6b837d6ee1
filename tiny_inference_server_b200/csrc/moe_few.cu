// The experts' products of few rows (a decode step), bfloat16: every expert that any row chose streams its matrices once.
//
// Bound by those bytes.  A dot product per (row, choice) and output element, as moe.cu does it, reads an expert's matrices
// once per row that chose it and spends a multiply-add per element and row on the CUDA cores; here 16 rows of a matrix are the
// rows of an mma.sync tile and up to 32 (row, choice) pairs of the expert its columns.  The summed index may run in any order
// that both operands agree on: a lane's 16 bytes of a matrix row (eight neighbouring elements) are its share of two products,
// and the same eight elements of its column's input row, so both come from global memory in 16-byte loads, as they lie.
// 8 rows of 1536, 16 experts of 1024 hidden elements, 3 a row: 21 + 23 us, 25 + 21 with a dot product per element (cold, under the
// profiler): so few rows seldom share an expert.  With more rows they do: a layer of 31 rows 47 us, 103 with dot products.
#include "common.cuh"

namespace {

constexpr int FEATURES = 16;             // matrix rows of a tile
constexpr int GROUPS = 4;                // column groups of eight pairs that one pass over a matrix serves
constexpr int FIRST_WARPS = 4, SHARES = 4;

__device__ __forceinline__ void mma_few(float (&c)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint4 load_once(const bf16* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory"); }
__device__ __forceinline__ float cluster_read(const float* mine, int rank) {
    unsigned at;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(at) : "r"((unsigned)__cvta_generic_to_shared(mine)), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];\n" : "=f"(v) : "r"(at) : "memory");
    return v;
}
__device__ __forceinline__ float few_act(float x, int kind) {
    if (kind == 0) { const float r = fmaxf(x, 0.f); return r * r; }
    if (kind == 1) return 0.5f * x * (1.f + tanhf(0.7978845608028654f * (x + 0.044715f * x * x * x)));
    return x / (1.f + expf(-x));
}

// The pairs that chose expert e, in order, by one warp; returns their number (the same in all lanes).
__device__ __forceinline__ int pairs_of(const int* chosen, int pairs, int e, int* list) {
    const int lane = threadIdx.x & 31;
    int count = 0;
    for (int base = 0; base < pairs; base += 32) {
        const bool mine = base + lane < pairs && chosen[base + lane] == e;
        const unsigned who = __ballot_sync(0xffffffffu, mine);
        if (mine) list[count + __popc(who & ((1u << lane) - 1u))] = base + lane;
        count += __popc(who);
    }
    __syncwarp();
    return count;
}

// acc[m][g] += W_m[16 rows] . X_g, G groups, over the blocks [from, to) of 32 elements; w[m]: this lane's place in its first row
// (rows lane / 4 and lane / 4 + 8, elements 8 (lane % 4)..), x[g]: in its column's input row.  The loads of AHEAD blocks are on
// their way together, inputs as well as weights: what the kernel before wrote comes from L2, as far away as the weights.
template <int MATS, int G, int AHEAD>
__device__ __forceinline__ void stream_groups(const bf16* const (&w)[MATS], size_t row8, const bf16* const (&x)[GROUPS], int from, int to,
                                              float (&acc)[MATS][GROUPS][4]) {
    for (int b0 = from; b0 < to; b0 += AHEAD) {
        uint4 a[AHEAD][MATS][2], v[AHEAD][G];
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
            const size_t at = (size_t)min(b0 + u, to - 1) * 32;
#pragma unroll
            for (int m = 0; m < MATS; ++m) { a[u][m][0] = load_once(w[m] + at); a[u][m][1] = load_once(w[m] + row8 + at); }
#pragma unroll
            for (int g = 0; g < G; ++g) v[u][g] = *reinterpret_cast<const uint4*>(x[g] + at);
        }
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
            if (b0 + u >= to) break;
#pragma unroll
            for (int g = 0; g < G; ++g)
#pragma unroll
                for (int m = 0; m < MATS; ++m) {
                    mma_few(acc[m][g], a[u][m][0].x, a[u][m][1].x, a[u][m][0].y, a[u][m][1].y, v[u][g].x, v[u][g].y);
                    mma_few(acc[m][g], a[u][m][0].z, a[u][m][1].z, a[u][m][0].w, a[u][m][1].w, v[u][g].z, v[u][g].w);
                }
        }
    }
}
template <int MATS>
__device__ __forceinline__ void stream(const bf16* const (&w)[MATS], size_t row8, const bf16* const (&x)[GROUPS], int groups, int from,
                                       int to, float (&acc)[MATS][GROUPS][4]) {
    if (groups == 1) stream_groups<MATS, 1, MATS == 2 ? 4 : 8>(w, row8, x, from, to, acc);
    else if (groups == 2) stream_groups<MATS, 2, MATS == 2 ? 3 : 5>(w, row8, x, from, to, acc);
    else stream_groups<MATS, GROUPS, 2>(w, row8, x, from, to, acc);
}

// hidden[pair][f] = gated(Wg[e][f] . x, Wu[e][f] . x) (MATS 2) or act(Wu[e][f] . x) (MATS 1), x the pair's row.  A CTA per (16
// hidden elements, expert), its warps a quarter of the sum each.
template <int MATS>
__global__ void __launch_bounds__(FIRST_WARPS * 32)
moe_few_first_kernel(const bf16* __restrict__ x, int ldx, const int* __restrict__ chosen, int pairs, int top, const bf16* __restrict__ w,
                     bf16* __restrict__ hidden, int d, int F, int act, GateForm gate, const float* __restrict__ in_weights) {
    extern __shared__ int list[];                           // [pairs]
    __shared__ float part[FIRST_WARPS][MATS][GROUPS][128];
    __shared__ int count_sh;
    pdl_launch_dependents();
    const int e = blockIdx.y, f0 = blockIdx.x * FEATURES;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, fr = lane >> 2, fc = lane & 3;
    pdl_wait();
    if (warp == 0) {
        const int c = pairs_of(chosen, pairs, e, list);
        if (lane == 0) count_sh = c;
    }
    __syncthreads();
    const int count = count_sh, blocks = d / 32;
    const bf16* we = w + ((size_t)e * MATS * F + f0 + fr) * d + fc * 8;
    for (int p0 = 0; p0 < count; p0 += 8 * GROUPS) {
        const int groups = min(GROUPS, (count - p0 + 7) / 8);
        const bf16* wm[MATS];
        const bf16* xg[GROUPS];
#pragma unroll
        for (int m = 0; m < MATS; ++m) wm[m] = we + (size_t)m * F * d;
#pragma unroll
        for (int g = 0; g < GROUPS; ++g) xg[g] = x + (size_t)(list[min(p0 + 8 * g + fr, count - 1)] / top) * ldx + fc * 8;
        float acc[MATS][GROUPS][4] = {};
        stream<MATS>(wm, (size_t)8 * d, xg, groups, blocks * warp / FIRST_WARPS, blocks * (warp + 1) / FIRST_WARPS, acc);
#pragma unroll
        for (int m = 0; m < MATS; ++m)
#pragma unroll
            for (int g = 0; g < GROUPS; ++g)
                *reinterpret_cast<float4*>(&part[warp][m][g][lane * 4]) = make_float4(acc[m][g][0], acc[m][g][1], acc[m][g][2], acc[m][g][3]);
        __syncthreads();
        for (int i = tid; i < groups * 128; i += FIRST_WARPS * 32) {
            // neighbouring threads: neighbouring hidden elements of one pair
            const int g = i / 128, n = i % 128 / 16, f = i % 16;
            const int at = ((f & 7) * 4 + (n >> 1)) * 4 + (f >> 3) * 2 + (n & 1), k = p0 + 8 * g + n;
            if (k >= count) continue;
            float v[MATS];
#pragma unroll
            for (int m = 0; m < MATS; ++m) {
                v[m] = 0.f;
#pragma unroll
                for (int s = 0; s < FIRST_WARPS; ++s) v[m] += part[s][m][g][at];
            }
            const int pair = list[k];
            const float iw = in_weights != nullptr ? in_weights[pair] : 1.f;
            hidden[(size_t)pair * F + f0 + f] = __float2bfloat16_rn(MATS == 2 ? gated_unit(v[0] * iw, v[MATS - 1] * iw, gate) : few_act(v[0] * iw, act));
        }
        __syncthreads();
    }
}

// out[r][c] = sum_k weights[r][k] * (Wd[e_k][c] . hidden[r * top + k]) (+ shared_gate[r] * shared[r][c]).  A cluster of 1, 2 or 4 CTAs
// per 16 output columns takes the chosen experts in turn, four warps an expert, a quarter of the sum each, and leaves the pairs'
// results in its CTAs' shared memory, where they are added up in the order of the choices whatever the size of the cluster.
template <int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 16 / WARPS)
moe_few_second_kernel(const bf16* __restrict__ hidden, const int* __restrict__ chosen, const float* __restrict__ weights, int pairs, int top,
                      const bf16* __restrict__ w, const bf16* __restrict__ shared, int lds, const float* __restrict__ shared_gate,
                      bf16* __restrict__ out, int d, int E, int F, int ctas) {
    extern __shared__ __align__(16) float smem[];
    float* part = smem;                                     // [SHARES][pairs][FEATURES]
    int* all = reinterpret_cast<int*>(part + (size_t)SHARES * pairs * FEATURES);        // [pairs] the choices
    int* list = all + pairs + (threadIdx.x >> 5) * pairs;   // [pairs] a warp's own
    unsigned* met = reinterpret_cast<unsigned*>(all + (WARPS + 1) * pairs);      // [E / 32] a bit for each chosen expert
    pdl_launch_dependents();
    const int rank = blockIdx.x % ctas, c0 = blockIdx.x / ctas * FEATURES;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, fr = lane >> 2, fc = lane & 3;
    const int blocks = F / 32, words = (E + 31) / 32, share = warp % SHARES;
    for (int i = tid; i < words; i += WARPS * 32) met[i] = 0;
    __syncthreads();
    pdl_wait();
    for (int i = tid; i < pairs; i += WARPS * 32) {
        const int e = chosen[i];
        all[i] = e;
        if (e >= 0 && e < E) atomicOr(&met[e >> 5], 1u << (e & 31));
    }
    __syncthreads();
    int turn = 0;                                           // chosen experts passed so far
    for (int word = 0; word < words; ++word)
        for (unsigned left = met[word]; left != 0; left &= left - 1, ++turn) {
            if (turn % ctas != rank || turn / ctas % (WARPS / SHARES) != warp / SHARES) continue;
            const int e = word * 32 + __ffs(left) - 1;
            const int count = pairs_of(all, pairs, e, list);
            for (int p0 = 0; p0 < count; p0 += 8 * GROUPS) {
                const int groups = min(GROUPS, (count - p0 + 7) / 8);
                const bf16* const wm[1] = {w + ((size_t)e * d + c0 + fr) * F + fc * 8};
                const bf16* xg[GROUPS];
#pragma unroll
                for (int g = 0; g < GROUPS; ++g) xg[g] = hidden + (size_t)list[min(p0 + 8 * g + fr, count - 1)] * F + fc * 8;
                float acc[1][GROUPS][4] = {};
                stream<1>(wm, (size_t)8 * F, xg, groups, blocks * share / SHARES, blocks * (share + 1) / SHARES, acc);
#pragma unroll
                for (int g = 0; g < GROUPS; ++g)
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int k = p0 + 8 * g + 2 * fc + (i & 1);
                        if (g < groups && k < count) part[((size_t)share * pairs + list[k]) * FEATURES + fr + (i >> 1) * 8] = acc[0][g][i];
                    }
            }
            __syncwarp();                                   // the list is written anew
        }
    if (ctas > 1) { cluster_arrive(); cluster_wait(); } else __syncthreads();
    for (int i = rank * WARPS * 32 + tid; i < pairs / top * FEATURES; i += ctas * WARPS * 32) {
        const int r = i / FEATURES, c = i % FEATURES;
        float acc = 0.f;
        for (int k = 0; k < top; ++k) {
            const int pair = r * top + k, e = all[pair];
            if (e < 0 || e >= E) continue;
            int home = __popc(met[e >> 5] & ((1u << (e & 31)) - 1u));        // the expert's turn, and with it its CTA
            for (int word = 0; word < e >> 5; ++word) home += __popc(met[word]);
            home %= ctas;
            float v = 0.f;
#pragma unroll
            for (int s = 0; s < SHARES; ++s) {
                const float* at = part + ((size_t)s * pairs + pair) * FEATURES + c;
                v += ctas > 1 ? cluster_read(at, home) : *at;
            }
            acc = fmaf(weights != nullptr ? weights[pair] : 1.f, v, acc);
        }
        if (shared != nullptr)
            acc = fmaf(shared_gate != nullptr ? shared_gate[r] : 1.f, __bfloat162float(shared[(size_t)r * lds + c0 + c]), acc);
        out[(size_t)r * d + c0 + c] = __float2bfloat16_rn(acc);
    }
    if (ctas > 1) { cluster_arrive(); cluster_wait(); }     // no CTA leaves while a neighbour reads its shared memory
}

}  // namespace

// The experts' products of n rows of `top` choices in bfloat16: x (n, d) with row stride ldx, w_gu (E, 2, F, d), or (E, F, d) with
// act >= 0 (units without a gate); w_down (E, d, F); hidden (n * top, F) scratch; weigh_input: a choice's weight multiplies its
// unit's input instead of its output.  d and F multiples of 32, rows and matrices on 16-byte boundaries, n * top at most 384.
TIS_API int tis_moe_few(const void* x, int ldx, const int* chosen, const float* weights, const void* w_gu, const void* w_down,
                        const void* shared, int lds, const float* shared_gate, void* out, void* hidden, int n, int d, int top, int E,
                        int F, int act, GateForm gate, int weigh_input, cudaStream_t stream) {
    if (n <= 0) return TIS_OK;
    const long long pairs = (long long)n * top;
    if (d <= 0 || F <= 0 || d % 32 || F % 32 || ldx % 8 || E <= 0 || E > 65535 || top <= 0 || pairs > 384 ||
        ((uintptr_t)x | (uintptr_t)w_gu | (uintptr_t)w_down | (uintptr_t)hidden) % 16) {
        tis_set_error("moe_few: width %d and hidden %d must be multiples of 32, %d rows of %d choices at most 384, operands aligned "
                      "(%d experts)", d, F, n, top, E);
        return TIS_BAD_SIZE;
    }
    const float* in_weights = weigh_input ? weights : nullptr;
    auto first = act >= 0 ? moe_few_first_kernel<1> : moe_few_first_kernel<2>;
    tis_launch(first, dim3(F / FEATURES, E), dim3(FIRST_WARPS * 32), sizeof(int) * (size_t)pairs, stream, (const bf16*)x, ldx, chosen,
               (int)pairs, top, (const bf16*)w_gu, (bf16*)hidden, d, F, act, gate, in_weights);
    const int st = tis_check_launch("moe_few_first");
    if (st != TIS_OK) return st;
    // Columns for fewer groups than SMs: 16 warps a CTA, one CTA an SM, and clusters of as many as the SMs hold.  For more: 8 warps, two
    // CTAs an SM (a second wave of a few CTAs would cost as much as the first).  us a layer, 64 experts of 512, width 1024, 4 rows of 6:
    // 37 alone, 29 as pairs, 40 as fours; 16 of 256, width 512, 32 rows of 3: 17.4, 14.6, 12.9; 16 of 1408, width 2048, 8 rows: 59, 64, 74;
    // 16 of 2048, width 3072, 4 rows: 99 with 16 warps a CTA, 87 with 8.
    const int columns = d / FEATURES, sms = 148;
    const int warps = columns <= sms ? 16 : 8, ctas = columns * 4 <= sms ? 4 : columns * 2 <= sms ? 2 : 1;
    auto second = warps == 16 ? moe_few_second_kernel<16> : moe_few_second_kernel<8>;
    const size_t smem = (sizeof(float) * SHARES * FEATURES + sizeof(int) * (warps + 1)) * (size_t)pairs + (size_t)(E + 31) / 32 * 4;
    if (smem > 48 * 1024) cudaFuncSetAttribute(second, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(columns * ctas);
    cfg.blockDim = dim3(warps * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int attrs = 0;
    if (ctas > 1) {
        attr[attrs].id = cudaLaunchAttributeClusterDimension;
        attr[attrs].val.clusterDim.x = ctas; attr[attrs].val.clusterDim.y = 1; attr[attrs++].val.clusterDim.z = 1;
    }
    if (tis_pdl_enabled()) {
        attr[attrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[attrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = attrs;
    cudaLaunchKernelEx(&cfg, second, (const bf16*)hidden, chosen, weigh_input ? (const float*)nullptr : weights, (int)pairs, top,
                       (const bf16*)w_down, (const bf16*)shared, lds, shared_gate, (bf16*)out, d, E, F, ctas);
    return tis_check_launch("moe_few_second");
}
