// Attention of single rows (a decode step) over the paged cache, for keys of TIS_KD and values of TIS_VD elements (compiled per
// pair of widths), with what windowed attention may ask for: a window or chunks, a distance bias or bounded scores, a sink,
// gates, and values that are the first elements of the key rows (SHARED).
//
// A CTA takes a row and a kv head with all its query heads (at most 16, one tile of mma.sync rows) and a share of the keys; the
// shares of a row are a thread-block cluster.  A fifth warp orders tiles of 64 keys by TMA boxes (64 elements x page rows,
// swizzled) STAGES ahead; each of four warps takes 16 keys of every tile, with a running maximum and sum of its own, and no
// barrier in the loop.  The warps' results are merged in shared memory, those of the cluster by reading the neighbours'
// shared memory, every CTA a part of the outputs: no second launch, no scratch in global memory.
// The shares are as many as keep all clusters resident at once (the device is asked how many it holds).
// Keys that the row does not see come from pages that may hold anything: their scores are masked and their value elements
// taken for zero.
// What bounds it: the chain from the page table through the first boxes to the merge.  8 rows at 4096 keys, 8 query heads of 128
// on each of 3 kv heads (50 MB): 37 + 7 us before (tiles of 64 keys by one of four warps in turn, shares merged by a second
// kernel), 21 us now (both cold, under the profiler).
#include "tc_common.cuh"

#ifndef TIS_KD
#define TIS_KD 128
#endif
#ifndef TIS_VD
#define TIS_VD 128
#endif

#if (TIS_KD % 64 == 0) && (TIS_VD % 64 == 0) && (TIS_KD <= 256) && (TIS_VD <= 128)

namespace {

using namespace tc;

constexpr int KD = TIS_KD, VD = TIS_VD, KEYS = 64, ROWS = 16, WARPS = 4;
constexpr int K_BLOCKS = KD / 64, V_BLOCKS = VD / 64, BLOCK_BYTES = KEYS * 128;
constexpr int QROW = KD + 8, PROW = VD + 2;
constexpr int STAGES = 3;
template <bool SHARED> __host__ __device__ constexpr int stage_bytes() { return (K_BLOCKS + (SHARED ? 0 : V_BLOCKS)) * BLOCK_BYTES; }
// the stages, which carry the warps' partial results afterwards; behind them the CTA's own result and the queries
template <bool SHARED> __host__ __device__ constexpr int tiles_bytes() {
    constexpr int a = STAGES * stage_bytes<SHARED>(), b = WARPS * ROWS * PROW * 4;
    return a > b ? a : b;
}
template <bool SHARED> constexpr int smem_bytes() { return tiles_bytes<SHARED>() + ROWS * PROW * 4 + ROWS * QROW * 2 + 1024; }

struct DecodeParams {
    const bf16* q; int ldq;
    const bf16* gate; int ldg, gate_per_head;
    bf16* out; int ldo;
    const int* block_table; int bt_stride, num_pages;
    const int* positions; const int* row_slot;
    int H, G, page_size, window;
    float scale;
    SoftCap cap;                     // bounds the raw scores (k 0: not)
    const float *r1, *r2;            // per query head (r1 null: no bias)
    const float* sink;               // per query head: exp(sink) is one more term of the softmax's denominator (null: none)
    int* fault;
};

__device__ __forceinline__ void ldmatrix_x4(unsigned (&r)[4], unsigned a) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
__device__ __forceinline__ void ldmatrix_x4_trans(unsigned (&r)[4], unsigned a) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ unsigned pack_bf16(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const unsigned*>(&v);
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory"); }
__device__ __forceinline__ float remote_f32(const float* mine, int rank) {
    unsigned at;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(at) : "r"(smem_u32(mine)), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];\n" : "=f"(v) : "r"(at) : "memory");
    return v;
}

template <bool SHARED>
__global__ void __launch_bounds__((WARPS + 1) * 32, 2)
window_attention_decode_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                               const DecodeParams p) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    float* own = reinterpret_cast<float*>(tiles + tiles_bytes<SHARED>());       // [ROWS][PROW]: out, maximum, sum
    bf16* qs = reinterpret_cast<bf16*>(own + ROWS * PROW);                      // [ROWS][QROW]
    __shared__ unsigned long long full[STAGES], empty[STAGES];
    __shared__ int abort_flag;
    __shared__ float top[ROWS][17], den[ROWS][17];          // per row and share of the keys: maximum, then factor; sum
    pdl_launch_dependents();
    const int split = blockIdx.x, splits = gridDim.x, kvh = blockIdx.y, row = blockIdx.z;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
    const int slot = p.row_slot[row], pos = p.positions[row];
    if (slot < 0) return;                                   // padding: the whole cluster leaves together
    const int gq = p.H / p.G;
    const int first = first_key(pos, p.window), begin = first & ~(KEYS - 1);
    const int all = (pos - begin) / KEYS + 1, per = (all + splits - 1) / splits;
    const int kt0 = min(all, split * per), count = min(all, kt0 + per) - kt0;
    if (tid == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], WARPS); }
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        prefetch_map(&map_k);
        if (!SHARED) prefetch_map(&map_v);
    }
    volatile int* abort = &abort_flag;
    float o[VD / 8][4], m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
#pragma unroll
    for (int n = 0; n < VD / 8; ++n) { o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f; }
    const int box = min(p.page_size, KEYS), ppt = KEYS / box;       // rows of a box, boxes of a tile side by side
    auto page_of = [&](int kt) -> int {
        if (lane >= ppt) return 0;
        const int key0 = begin + kt * KEYS + lane * box;
        if (key0 > pos || key0 + box <= first) return 0;    // no key of it is seen: any page will do
        const int pg = p.block_table[(size_t)slot * p.bt_stride + key0 / p.page_size];
        if (pg < 0 || pg >= p.num_pages) { atomicExch(p.fault, 5); return 0; }
        return pg;
    };
    int page = warp == WARPS && count > 0 ? page_of(kt0) : 0;
    __syncthreads();
    pdl_wait();
    if (warp == WARPS) {
        for (int i = 0; i < count; ++i) {
            const int s = i % STAGES, now = page;
            page = i + 1 < count ? page_of(kt0 + i + 1) : 0;
            int got = 1;
            if (lane == 0) got = mbar_wait(&empty[s], ((i / STAGES) & 1) ^ 1, abort, p.fault, 6) ? 1 : 0;
            got = __shfl_sync(0xffffffffu, got, 0);
            if (!got) break;
            if (lane == 0) mbar_arrive_expect_tx(&full[s], stage_bytes<SHARED>());
            __syncwarp();
            if (lane < ppt) {
                unsigned char* dst = tiles + s * stage_bytes<SHARED>() + lane * box * 128;
                const int y = kvh * p.page_size + (begin + (kt0 + i) * KEYS + lane * box) % p.page_size;
                for (int b = 0; b < K_BLOCKS; ++b) tma_load_3d(dst + b * BLOCK_BYTES, &map_k, b * 64, y, now, &full[s]);
                if (!SHARED)
                    for (int b = 0; b < V_BLOCKS; ++b) tma_load_3d(dst + (K_BLOCKS + b) * BLOCK_BYTES, &map_v, b * 64, y, now, &full[s]);
            }
        }
    } else {
        for (int i = tid; i < ROWS * (KD / 8); i += WARPS * 32) {
            const int r = i / (KD / 8), c = i % (KD / 8);
            *reinterpret_cast<uint4*>(qs + r * QROW + c * 8) = r < gq ?
                *reinterpret_cast<const uint4*>(p.q + (size_t)row * p.ldq + (size_t)(kvh * gq + r) * KD + c * 8) : make_uint4(0u, 0u, 0u, 0u);
        }
        asm volatile("bar.sync 1, 128;\n" ::: "memory");
        unsigned qf[KD / 16][4];
#pragma unroll
        for (int kk = 0; kk < KD / 16; ++kk)
            ldmatrix_x4(qf[kk], smem_u32(qs + ((lane & 7) + 8 * ((lane >> 3) & 1)) * QROW + kk * 16 + 8 * (lane >> 4)));
        float b1[2] = {0.f, 0.f}, b2[2] = {0.f, 0.f};
        if (p.r1 != nullptr) {
#pragma unroll
            for (int h = 0; h < 2; ++h)
                if (g + 8 * h < gq) { b1[h] = p.r1[kvh * gq + g + 8 * h]; b2[h] = p.r2[kvh * gq + g + 8 * h]; }
        }
        // where this lane's rows of an 8 x 8 block lie: of the keys (a key a row), of the values (transposed)
        const int k_row = warp * 16 + (lane & 7) + 8 * (lane >> 4), k_chunk = (lane >> 3) & 1;
        const int v_row = warp * 16 + (lane & 7) + 8 * ((lane >> 3) & 1), v_chunk = lane >> 4;
        for (int i = 0; i < count; ++i) {
            const int s = i % STAGES;
            if (!__all_sync(0xffffffffu, mbar_wait(&full[s], (i / STAGES) & 1, abort, p.fault, 6))) break;
            const unsigned ks = smem_u32(tiles + s * stage_bytes<SHARED>());
            const unsigned vs = SHARED ? ks : ks + K_BLOCKS * BLOCK_BYTES;
            const int j0 = begin + (kt0 + i) * KEYS + warp * 16;
            float sc[2][4] = {};
#pragma unroll
            for (int kk = 0; kk < KD / 16; ++kk) {
                unsigned b[4];
                ldmatrix_x4(b, ks + (kk >> 2) * BLOCK_BYTES + k_row * 128 + ((((kk & 3) * 2 + k_chunk) ^ (k_row & 7)) << 4));
                mma_bf16(sc[0], qf[kk], b[0], b[1]);
                mma_bf16(sc[1], qf[kk], b[2], b[3]);
            }
            if (p.cap.k != 0.f) {
#pragma unroll
                for (int n = 0; n < 2; ++n)
#pragma unroll
                    for (int e = 0; e < 4; ++e) sc[n][e] = soft_capped(sc[n][e], p.cap);
            }
            float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int j = j0 + n * 8 + 2 * t4 + (e & 1);
                    float v = sc[n][e] * p.scale;
                    if (p.r1 != nullptr) v -= b1[e >> 1] * __logf(fmaf(b2[e >> 1], (float)(pos - j), 1.f));
                    sc[n][e] = j >= first && j <= pos ? v : -INFINITY;
                    mx[e >> 1] = fmaxf(mx[e >> 1], sc[n][e]);
                }
            float corr[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 1));
                mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 2));
                const float m_new = fmaxf(m[h], mx[h]);
                corr[h] = m[h] == -INFINITY ? 0.f : __expf(m[h] - m_new);
                m[h] = m_new;
                l[h] *= corr[h];
            }
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float pv = sc[n][e] == -INFINITY ? 0.f : __expf(sc[n][e] - m[e >> 1]);
                    sc[n][e] = pv;
                    l[e >> 1] += pv;
                }
#pragma unroll
            for (int n = 0; n < VD / 8; ++n) {
                o[n][0] *= corr[0]; o[n][1] *= corr[0];
                o[n][2] *= corr[1]; o[n][3] *= corr[1];
            }
            // out += P V; elements of keys that are not seen are taken for zero
            unsigned pa[4];
#pragma unroll
            for (int a = 0; a < 4; ++a) pa[a] = pack_bf16(sc[a >> 1][(a & 1) * 2], sc[a >> 1][(a & 1) * 2 + 1]);
            unsigned keep[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int j = j0 + 2 * t4 + 8 * h;
                keep[h] = (j >= first && j <= pos ? 0x0000ffffu : 0u) | (j + 1 >= first && j + 1 <= pos ? 0xffff0000u : 0u);
            }
#pragma unroll
            for (int n2 = 0; n2 < VD / 16; ++n2) {
                unsigned b[4];
                ldmatrix_x4_trans(b, vs + (n2 >> 2) * BLOCK_BYTES + v_row * 128 + ((((n2 & 3) * 2 + v_chunk) ^ (v_row & 7)) << 4));
                mma_bf16(o[2 * n2], pa, b[0] & keep[0], b[1] & keep[1]);
                mma_bf16(o[2 * n2 + 1], pa, b[2] & keep[0], b[3] & keep[1]);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[s]);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            l[h] += __shfl_xor_sync(0xffffffffu, l[h], 1);
            l[h] += __shfl_xor_sync(0xffffffffu, l[h], 2);
        }
    }
    __syncthreads();                                        // every tile has been read: the stages carry the warps' results
    if (*abort) {
        // a wait ran out: give boxes that may still be on their way time to land before the stages carry anything else, and
        // before the shared memory is given up
        for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    }
    float* part = reinterpret_cast<float*>(tiles);          // [WARPS][ROWS][PROW]
    if (warp < WARPS) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float* dst = part + (warp * ROWS + g + 8 * h) * PROW;
#pragma unroll
            for (int n = 0; n < VD / 8; ++n)
                *reinterpret_cast<float2*>(dst + n * 8 + 2 * t4) = make_float2(o[n][2 * h], o[n][2 * h + 1]);
            if (t4 == 0) { dst[VD] = m[h]; dst[VD + 1] = l[h]; }
        }
    }
    __syncthreads();
    for (int i = tid; i < gq * VD; i += blockDim.x) {
        const int r = i / VD, c = i - r * VD;
        float mm = -INFINITY, num = 0.f, sum = 0.f;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) mm = fmaxf(mm, part[(w * ROWS + r) * PROW + VD]);
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
            const float* src = part + (w * ROWS + r) * PROW;
            const float f = src[VD] == -INFINITY ? 0.f : __expf(src[VD] - mm);
            num = fmaf(src[c], f, num);
            sum = fmaf(src[VD + 1], f, sum);
        }
        own[r * PROW + c] = num;
        if (c == 0) { own[r * PROW + VD] = mm; own[r * PROW + VD + 1] = sum; }
    }
    if (splits > 1) {
        cluster_arrive();
        cluster_wait();
    } else {
        __syncthreads();
    }
    for (int i = tid; i < gq * splits; i += blockDim.x) {
        const int r = i / splits, s = i - r * splits;
        top[r][s] = splits > 1 ? remote_f32(own + r * PROW + VD, s) : own[r * PROW + VD];
        den[r][s] = splits > 1 ? remote_f32(own + r * PROW + VD + 1, s) : own[r * PROW + VD + 1];
    }
    __syncthreads();
    if (tid < gq) {                                         // a row's factors, with its sum and the sink's term in them
        const float sk = p.sink != nullptr ? p.sink[kvh * gq + tid] : -INFINITY;
        float mm = sk, sum = 0.f;
        for (int s = 0; s < splits; ++s) mm = fmaxf(mm, top[tid][s]);
        for (int s = 0; s < splits; ++s) {
            top[tid][s] = top[tid][s] == -INFINITY ? 0.f : __expf(top[tid][s] - mm);
            sum = fmaf(den[tid][s], top[tid][s], sum);
        }
        if (sk != -INFINITY) sum += __expf(sk - mm);
        const float inv = sum > 0.f ? 1.f / sum : 0.f;
        for (int s = 0; s < splits; ++s) top[tid][s] *= inv;
    }
    __syncthreads();
    for (int i = split * blockDim.x + tid; i < gq * VD; i += splits * blockDim.x) {
        const int r = i / VD, c = i - r * VD;
        float x = 0.f;
        if (splits > 1) {
#pragma unroll 8
            for (int s = 0; s < splits; ++s) x = fmaf(remote_f32(own + r * PROW + c, s), top[r][s], x);
        } else {
            x = own[r * PROW + c] * top[r][0];
        }
        const int head = kvh * gq + r;
        if (p.gate != nullptr)
            x = x / (1.f + __expf(-__bfloat162float(p.gate[(size_t)row * p.ldg + (p.gate_per_head ? head : head * VD + c)])));
        p.out[(size_t)row * p.ldo + (size_t)head * VD + c] = __float2bfloat16_rn(x);
    }
    if (splits > 1) {                                       // nobody's memory goes while a neighbour reads it
        cluster_arrive();
        cluster_wait();
    }
}

template <bool SHARED>
int resident_clusters(int splits) {
    auto kernel = window_attention_decode_kernel<SHARED>;
    constexpr int smem = smem_bytes<SHARED>();
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(splits, 1, 1);
    cfg.blockDim = dim3((WARPS + 1) * 32);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = splits; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) { cudaGetLastError(); return 0; }
    return n;
}

template <bool SHARED>
int launch_decode(const CUtensorMap& mk, const CUtensorMap& mv, const DecodeParams& p, int rows, int splits, cudaStream_t stream) {
    auto kernel = window_attention_decode_kernel<SHARED>;
    constexpr int smem = smem_bytes<SHARED>();
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess ||
        cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
        return tis_check_launch("window_attention_decode (attributes)");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(splits, p.G, rows);
    cfg.blockDim = dim3((WARPS + 1) * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = splits; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = tis_pdl_enabled() ? 2 : 1;
    cudaLaunchKernelEx(&cfg, kernel, mk, mv, p);
    return tis_check_launch("window_attention_decode");
}

}  // namespace

// Whether this pair of widths has the kernel (1), also with values that are the first elements of the key rows (3).
TIS_API int tis_window_attention_decode_forms() { return TIS_KD >= TIS_VD ? 3 : 1; }

// How many clusters of `splits` CTAs the device holds at once.
TIS_API int tis_window_attention_decode_clusters(int shared, int splits) {
    if (!shared) return resident_clusters<false>(splits);
#if TIS_KD >= TIS_VD
    return resident_clusters<true>(splits);
#else
    return 0;
#endif
}

// Attention of `rows` single rows.  At most 16 query heads a kv head; `splits` 1, 2, 4, 8 or 16 shares of the keys; operands as
// for tis_window_attention_tc, any sign of the scale.
TIS_API int tis_window_attention_decode(const void* q, int ldq, const void* gate, int ldg, int gate_per_head, void* out, int ldo,
                                        const void* k_pages, size_t k_page_stride, const void* v_pages, size_t v_page_stride,
                                        int shared, const int* block_table, int bt_stride, int num_pages, const int* positions,
                                        const int* row_slot, int rows, int H, int G, int page_size, int window, float scale,
                                        float softcap, const float* r1, const float* r2, const float* sink, int splits, int* fault,
                                        cudaStream_t stream) {
    if (rows <= 0) return TIS_OK;
    if ((page_size != 16 && page_size != 32 && page_size != 64 && page_size != 128) || H <= 0 || G <= 0 || H % G || H / G > ROWS ||
        rows > 65535 || G > 65535 || ldq % 8 || k_page_stride % 8 || v_page_stride % 8 ||
        ((uintptr_t)q | (uintptr_t)k_pages | (uintptr_t)v_pages) % 16 || (r1 != nullptr && (softcap > 0.f || window < 0)) ||
        (splits != 1 && splits != 2 && splits != 4 && splits != 8 && splits != 16) ||
        !((tis_window_attention_decode_forms() >> (shared ? 1 : 0)) & 1)) {
        tis_set_error("window_attention_decode: %d query heads on %d, page size %d, %d rows, %d shares of the keys, row stride %d, or "
                      "operands that are not aligned", H, G, page_size, rows, splits, ldq);
        return TIS_BAD_SIZE;
    }
    CUtensorMap mk, mv;
    const int box = page_size < KEYS ? page_size : KEYS;
    if (!page_map(k_pages, KD, G * page_size, num_pages, KD, k_page_stride, box, &mk)) return TIS_CUDA_ERROR;
    if (shared) mv = mk;
    else if (!page_map(v_pages, VD, G * page_size, num_pages, VD, v_page_stride, box, &mv)) return TIS_CUDA_ERROR;
    DecodeParams p;
    p.q = (const bf16*)q; p.ldq = ldq;
    p.gate = (const bf16*)gate; p.ldg = ldg; p.gate_per_head = gate_per_head;
    p.out = (bf16*)out; p.ldo = ldo;
    p.block_table = block_table; p.bt_stride = bt_stride; p.num_pages = num_pages;
    p.positions = positions; p.row_slot = row_slot;
    p.H = H; p.G = G; p.page_size = page_size; p.window = window;
    p.scale = scale;
    p.cap = soft_cap(softcap, scale);
    p.r1 = r1; p.r2 = r2; p.sink = sink; p.fault = fault;
    if (!shared) return launch_decode<false>(mk, mv, p, rows, splits, stream);
#if TIS_KD >= TIS_VD
    return launch_decode<true>(mk, mv, p, rows, splits, stream);
#else
    return TIS_BAD_SIZE;
#endif
}

#else

TIS_API int tis_window_attention_decode_forms() { return 0; }
TIS_API int tis_window_attention_decode_clusters(int, int) { return 0; }

TIS_API int tis_window_attention_decode(const void*, int, const void*, int, int, void*, int, const void*, size_t, const void*,
                                        size_t, int, const int*, int, int, const int*, const int*, int, int, int, int, int, float,
                                        float, const float*, const float*, const float*, int, int*, cudaStream_t) {
    tis_set_error("window_attention_decode: built for widths it does not take");
    return TIS_BAD_SIZE;
}

#endif
