// Matrix products with many rows on the fifth-generation tensor cores:
// y (M x N) = x (M x K) . W (K x N), bfloat16 in, float32 accumulation — the projections of
// prompt portions.  Epilogues: plain bfloat16 store, or gating of [32 gate | 32 up]
// column blocks (the result then has N/2 columns), so the gate/up product never goes to memory.
//
// Persistent CTAs walk output tiles.  With CG = 2 two CTAs (a cluster, two SMs) share a tile of 256 rows x BN columns:
// each brings its own 128 rows of x and half of the columns of W, the products (cta_group::2, issued by the first CTA)
// read both halves, and each CTA's tensor memory holds its own 128 rows.  A tile of 256 x 256 then costs 64 bytes a cycle
// and SM from L2, where a tile of 128 x 256 by one CTA (CG = 1, for few rows) costs 96.
// Three roles, specialised by warp:
//   warp 0   one lane orders the operand tiles from the TMA engine (cp.async.bulk.tensor.2d
//            with the 128-byte swizzle; rows beyond M, columns beyond N and K beyond its end
//            are filled with zeros by the engine) into a ring of shared-memory stages; both
//            CTAs' copies count on the first one's barrier;
//   warp 1   owns the tensor memory (tcgen05.alloc) and, in the first CTA, one lane issues
//            tcgen05.mma: x tile as the K-major operand, W tile as the MN-major operand (W lies
//            (K, N) in memory, N contiguous, and is used as it is), accumulator in tensor memory;
//            tcgen05.commit hands a stage back to both CTAs' warps 0 and a finished accumulator
//            to both epilogues;
//   warps 2-5 read the accumulator (tcgen05.ld, one row per thread), apply the epilogue and
//            store.  The accumulator is double-buffered: the epilogue of one tile runs under
//            the products of the next.
// All hand-offs are mbarriers; every wait is bounded and a wait that runs out sets the fault
// word, lets every role leave its loop, and the tensor memory is freed before the CTA ends;
// the two CTAs of a cluster end together.
// A stage of 128 along K takes its products 1024 cycles (BN = 256) and some 300 to hand over; with wide tiles the operands from L2
// bound it.  Measured on a B200, us, the library's product and the gating kernel / this: 2048 x 1536 x 8192 49.7 / 40.2 (one CTA a tile,
// a look at a barrier 200 cycles and the division operator in the gating before: 52), 2048 x 3072 x 16384 160 / 138, 1024 x 1536 x
// 8192 27.7 / 23.7, 128 x 1536 x 8192 9.9 / 9.3.  Plain products it loses (2048 x 1536 x 2304 12.1 / 16.2, 2048 x 4096 x 1536
// 20.1 / 24.8, 2048 x 3072 x 12352 102 / 109): the library splits their sums, and its clusters fetch a tile once for several CTAs.
#include "tc_common.cuh"

namespace {

using namespace tc;

constexpr int BM = 128;                     // rows of a CTA
constexpr int BK = 64;                      // 64 bfloat16 = one 128-byte swizzle row
constexpr int NTH = 192;
constexpr int A_BYTES = BM * BK * 2;        // 16 KB
constexpr int BOX_B_BYTES = 64 * BK * 2;    // a W box: 64 rows of K x 64 columns = 8 KB

enum { EPI_STORE = 0, EPI_SWIGLU = 1 };

struct TcParams {
    bf16* out; int ldo;
    int M, N, K;
    int tiles_m, tiles_n;
    int* fault;
    GateForm gate;              // EPI_SWIGLU: the form of the gating
};

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm("mov.u32 %0, %cluster_ctarank;\n" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_meet() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
// the address of the same variable in the cluster's first CTA
__device__ __forceinline__ unsigned in_first(unsigned addr) {
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, 0;\n" : "=r"(r) : "r"(addr));
    return r;
}
// a box for this CTA whose bytes count on a barrier of the cluster's first CTA
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, int x, int y, unsigned bar) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n"
                 ::"r"(smem_u32(dst)), "l"(reinterpret_cast<unsigned long long>(map)), "r"(bar), "r"(x), "r"(y) : "memory");
}
template <int CG> __device__ __forceinline__ void product(unsigned d, unsigned long long a, unsigned long long b, unsigned idesc, unsigned more) {
    if constexpr (CG == 1) umma(d, a, b, idesc, more);
    else
        asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
                     "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n"
                     ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(more) : "memory");
}
template <int CG> __device__ __forceinline__ void commit(unsigned long long* bar) {
    if constexpr (CG == 1) umma_commit(bar);
    else
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n"
                     ::"r"(smem_u32(bar)), "h"((unsigned short)3) : "memory");
}

template <int CG, int BN> struct Tile {
    static constexpr int COLS = BN / CG;                        // of W that a CTA brings
    static constexpr int BOXES = (COLS + 63) / 64;
    static constexpr int SUB = CG == 1 && BN == 256 ? 1 : 2;    // steps of 64 along K a stage: a hand-over takes some 300 cycles
    static constexpr int STEP_BYTES = A_BYTES + BOXES * BOX_B_BYTES;
    static constexpr int STAGE_BYTES = SUB * STEP_BYTES;
    static constexpr int STAGES = 196608 / STAGE_BYTES < 8 ? 196608 / STAGE_BYTES : 8;
    static constexpr int ACC_COLS = BN > 128 ? 256 : (BN > 64 ? 128 : 64);
    static constexpr unsigned TMEM_COLS = 2 * ACC_COLS;         // two accumulators of BN float32 columns (a power of two)
};

template <int CG, int BN, int EPI>
__device__ __forceinline__ void gemm_tc_body(const CUtensorMap& map_a, const CUtensorMap& map_b, const TcParams& p) {
    typedef Tile<CG, BN> T;
    constexpr int STAGES = T::STAGES, STAGE_BYTES = T::STAGE_BYTES;
    constexpr unsigned IDESC = instr_desc(BM * CG, BN, true);

    extern __shared__ unsigned char smem_raw[];
    // operand tiles at 1024-byte boundaries: the swizzle is a function of the address
    unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ unsigned long long full[STAGES], empty[STAGES], acc_full[2], acc_empty[2];
    __shared__ unsigned tmem_base_slot;
    __shared__ int abort_flag;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = CG == 2 ? (int)cluster_rank() : 0, group = blockIdx.x / CG, groups = gridDim.x / CG;
    const int num_tiles = p.tiles_m * p.tiles_n;
    const int kt_count = (p.K + T::SUB * BK - 1) / (T::SUB * BK);

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 4 * CG); }
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        prefetch_map(&map_a);
        prefetch_map(&map_b);
    }
    if (warp == 1) {
        if constexpr (CG == 1) tmem_alloc(&tmem_base_slot, T::TMEM_COLS);
        else {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n"
                         ::"r"(smem_u32(&tmem_base_slot)), "r"(T::TMEM_COLS) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::: "memory");
        }
    }
    fence_before();
    __syncthreads();
    if constexpr (CG == 2) cluster_meet();                // the other CTA's barriers are there
    fence_after();
    pdl_launch_dependents();                              // (not before this CTA has its tensor memory: the next kernel may want some)
    const unsigned tmem_base = tmem_base_slot;
    volatile int* abort = &abort_flag;
    pdl_wait();                                           // x is the output of the kernel before

    if (warp == 0) {
        int it = 0;
        bool ok = true;
        for (int tile = group; tile < num_tiles && ok; tile += groups) {
            const int m0 = (tile % p.tiles_m * CG + rank) * BM, n0 = tile / p.tiles_m * BN + rank * T::COLS;
            for (int kt = 0; kt < kt_count; ++kt, ++it) {
                const int s = it % STAGES;
                if (!__all_sync(0xffffffffu, mbar_wait(&empty[s], ((it / STAGES) & 1) ^ 1, abort, p.fault, 5))) { ok = false; break; }
                if (elect_one()) {
                    unsigned char* a = tiles + s * STAGE_BYTES;
                    if (rank == 0) mbar_arrive_expect_tx(&full[s], CG * STAGE_BYTES);
                    const unsigned bar = CG == 2 ? in_first(smem_u32(&full[s])) : 0u;
#pragma unroll
                    for (int sub = 0; sub < T::SUB; ++sub, a += T::STEP_BYTES) {
                        const int k = (kt * T::SUB + sub) * BK;
                        if constexpr (CG == 1) tma_load_2d(a, &map_a, k, m0, &full[s]);
                        else tma_load_2d_pair(a, &map_a, k, m0, bar);
#pragma unroll
                        for (int j = 0; j < T::BOXES; ++j) {
                            if constexpr (CG == 1) tma_load_2d(a + A_BYTES + j * BOX_B_BYTES, &map_b, n0 + j * 64, k, &full[s]);
                            else tma_load_2d_pair(a + A_BYTES + j * BOX_B_BYTES, &map_b, n0 + j * 64, k, bar);
                        }
                    }
                }
                __syncwarp();
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {
            // descriptors differ from the first stage's in the start address only (units of 16 bytes)
            const unsigned long long a0 = smem_desc(smem_u32(tiles), 16, 1024), b0 = smem_desc(smem_u32(tiles) + A_BYTES, BOX_B_BYTES, 1024);
            int it = 0, acc_it = 0;
            bool ok = true;
            for (int tile = group; tile < num_tiles && ok; tile += groups, ++acc_it) {
                const int b = acc_it & 1;
                if (!__all_sync(0xffffffffu, mbar_wait(&acc_empty[b], ((acc_it >> 1) & 1) ^ 1, abort, p.fault, 5))) break;
                fence_after();
                const unsigned d = tmem_base + b * T::ACC_COLS;
                for (int kt = 0; kt < kt_count; ++kt, ++it) {
                    const int s = it % STAGES;
                    if (!__all_sync(0xffffffffu, mbar_wait(&full[s], (it / STAGES) & 1, abort, p.fault, 5))) { ok = false; break; }
                    fence_after();
                    if (elect_one()) {
#pragma unroll
                        for (int kk = 0; kk < T::SUB * BK / 16; ++kk) {
                            const unsigned at = (unsigned)(s * STAGE_BYTES + kk / 4 * T::STEP_BYTES) >> 4;
                            // x: 16 elements of K further = 32 bytes inside the swizzled 128-byte row;
                            // W: 16 rows of K further = two groups of eight 128-byte rows
                            product<CG>(d, a0 + at + kk % 4 * 2, b0 + at + kk % 4 * 128, IDESC, (kt | kk) != 0);
                        }
                        commit<CG>(&empty[s]);            // the stage is free when these products have read it
                        if (kt == kt_count - 1) commit<CG>(&acc_full[b]);
                    }
                    __syncwarp();
                }
            }
        }
    } else {
        const int quarter = warp & 3;                     // the 32 lanes of tensor memory this warp may read
        int acc_it = 0;
        for (int tile = group; tile < num_tiles; tile += groups, ++acc_it) {
            const int b = acc_it & 1;
            const int m0 = (tile % p.tiles_m * CG + rank) * BM, n0 = tile / p.tiles_m * BN;
            if (!__all_sync(0xffffffffu, mbar_wait(&acc_full[b], (acc_it >> 1) & 1, abort, p.fault, 5))) break;
            fence_after();
            const int row = m0 + quarter * 32 + lane;
            const unsigned taddr = tmem_base + ((unsigned)(quarter * 32) << 16) + b * T::ACC_COLS;
            if constexpr (EPI == EPI_STORE) {
#pragma unroll 1
                for (int c = 0; c < BN / 32; ++c) {
                    float v[32];
                    tmem_ld32(taddr + c * 32, v);
                    const int col = n0 + c * 32;
                    if (row < p.M) {
                        bf16* o = p.out + (size_t)row * p.ldo + col;
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            if (col + q * 8 < p.N) store8(o + q * 8, v + q * 8);
                    }
                    __syncwarp();
                }
            } else {
#pragma unroll 1
                for (int c = 0; c < BN / 64; ++c) {
                    float g[32], u[32];
                    tmem_ld32_issue(taddr + c * 64, g);
                    tmem_ld32_issue(taddr + c * 64 + 32, u);
                    tmem_ld_wait();
                    tmem_ld_arrived(g);
                    tmem_ld_arrived(u);
#pragma unroll
                    for (int i = 0; i < 32; ++i) g[i] = gated_unit_epilogue(g[i], u[i], p.gate);
                    if (row < p.M && n0 + c * 64 < p.N) {
                        bf16* o = p.out + (size_t)row * p.ldo + (n0 >> 1) + c * 32;
#pragma unroll
                        for (int q = 0; q < 4; ++q) store8(o + q * 8, g + q * 8);
                    }
                    __syncwarp();
                }
            }
            fence_before();
            __syncwarp();
            if (lane == 0) {
                if constexpr (CG == 1) mbar_arrive(&acc_empty[b]);
                else asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];\n" ::"r"(in_first(smem_u32(&acc_empty[b]))) : "memory");
            }
        }
    }
    __syncwarp();

    if (*abort) {
        // a wait ran out: give copies that may still be in flight time to land before the
        // shared memory is given up
        for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    }
    fence_before();
    __syncthreads();
    if constexpr (CG == 2) cluster_meet();                // the products that read this CTA's operands, and arrivals, are done
    if (warp == 1) {
        fence_after();
        if constexpr (CG == 1) tmem_free(tmem_base, T::TMEM_COLS);
        else
            asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(T::TMEM_COLS) : "memory");
    }
}

template <int BN, int EPI>
__global__ void __launch_bounds__(NTH, 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const TcParams p) {
    gemm_tc_body<1, BN, EPI>(map_a, map_b, p);
}
template <int BN, int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(NTH, 1)
gemm_tc_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const TcParams p) {
    gemm_tc_body<2, BN, EPI>(map_a, map_b, p);
}

// ---- host side ----------------------------------------------------------------------------

template <int CG, int BN, int EPI>
int launch(const CUtensorMap& ma, const CUtensorMap& mb, TcParams p, cudaStream_t stream) {
    constexpr int smem = Tile<CG, BN>::STAGES * Tile<CG, BN>::STAGE_BYTES + 1024;
    void (*kernel)(CUtensorMap, CUtensorMap, TcParams);
    if constexpr (CG == 1) kernel = gemm_tc_kernel<BN, EPI>;
    else kernel = gemm_tc_pair_kernel<BN, EPI>;
    static bool configured = false;
    if (!configured) {
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
            return tis_check_launch("gemm_tc (shared memory)");
        configured = true;
    }
    p.tiles_m = (p.M + BM * CG - 1) / (BM * CG);
    p.tiles_n = (p.N + BN - 1) / BN;
    const int tiles = p.tiles_m * p.tiles_n, groups = sm_count() / CG;
    tis_launch(kernel, dim3((tiles < groups ? tiles : groups) * CG), dim3(NTH), (size_t)smem, stream, ma, mb, p);
    return tis_check_launch("gemm_tc");
}

template <int EPI> int launch_shape(int shape, const CUtensorMap& ma, const CUtensorMap& mb, const TcParams& p, cudaStream_t stream) {
    switch (shape) {
        case 0: return launch<2, 256, EPI>(ma, mb, p, stream);
        case 1: return launch<2, 192, EPI>(ma, mb, p, stream);
        case 2: return launch<2, 128, EPI>(ma, mb, p, stream);
        case 3: return launch<1, 256, EPI>(ma, mb, p, stream);
        case 4: return launch<1, 128, EPI>(ma, mb, p, stream);
        default: return launch<1, 64, EPI>(ma, mb, p, stream);
    }
}

}  // namespace

// y = x . W on the tcgen05 tensor cores.  x (M x K, row stride ldx), W (K x N, row stride ldw), out (M x N, or
// M x N/2 with epi = 1), all bfloat16, strides in elements.  Refuses what the
// TMA engine cannot address: K, N and the strides must be multiples of 8 elements and the
// pointers 16-byte aligned; with epi = 1, N must be a multiple of 64.  shape -1: the kernel's own choice of tile (tests ask
// for the others).
TIS_API int tis_gemm_tc(const void* x, int ldx, const void* w, int ldw, void* out, int ldo, int M, int N, int K,
                        int epi, GateForm gate, int shape, int* fault, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return TIS_OK;
    if (K <= 0 || (K % 8) || (N % 8) || (ldx % 8) || (ldw % 8) || (ldo % 8) ||
        (reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(out)) % 16) {
        tis_set_error("gemm_tc: M %d N %d K %d strides %d %d %d: K, N and the strides must be multiples of 8 and the "
                      "pointers 16-byte aligned", M, N, K, ldx, ldw, ldo);
        return TIS_BAD_SIZE;
    }
    if (epi != EPI_STORE && epi != EPI_SWIGLU) {
        tis_set_error("gemm_tc: unknown epilogue %d", epi);
        return TIS_BAD_SIZE;
    }
    if (epi == EPI_SWIGLU && (N % 64)) {
        tis_set_error("gemm_tc: the SwiGLU epilogue takes N a multiple of 64, got %d", N);
        return TIS_BAD_SIZE;
    }
    CUtensorMap ma, mb;
    if (!tensor_map(x, K, M, ldx, BM, true, &ma) || !tensor_map(w, N, K, ldw, BK, true, &mb)) return TIS_CUDA_ERROR;
    TcParams p;
    p.out = static_cast<bf16*>(out);
    p.ldo = ldo;
    p.M = M; p.N = N; p.K = K;
    p.tiles_m = p.tiles_n = 0;
    p.fault = fault;
    p.gate = gate;
    if (shape < 0) {
        // The tile that needs the least time by a simple count: rounds of tiles over the SMs times the cycles of a tile's
        // products (or of its operands from L2, 60 bytes a cycle and SM), and the last tile's way out
        static const int cg[6] = {2, 2, 2, 1, 1, 1}, bn[6] = {256, 192, 128, 256, 128, 64};
        const int sms = sm_count(), kt = (K + BK - 1) / BK;
        long long best = -1;
        for (int i = 0; i < 6; ++i) {
            const long long tiles = (long long)((M + BM * cg[i] - 1) / (BM * cg[i])) * ((N + bn[i] - 1) / bn[i]);
            const int boxes = (bn[i] / cg[i] + 63) / 64, feed = (A_BYTES + boxes * BOX_B_BYTES) / 60;
            const long long rounds = (tiles * cg[i] + sms - 1) / sms;
            const long long cost = rounds * kt * (2 * bn[i] > feed ? 2 * bn[i] : feed) + 12 * bn[i];
            if (best < 0 || cost < best) { best = cost; shape = i; }
        }
    }
    if (epi == EPI_STORE) return launch_shape<EPI_STORE>(shape, ma, mb, p, stream);
    return launch_shape<EPI_SWIGLU>(shape, ma, mb, p, stream);
}
