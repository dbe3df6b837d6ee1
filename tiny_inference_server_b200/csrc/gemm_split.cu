// Matrix products of 32-bit operands on the fifth-generation tensor cores: y (M x N) = x (M x K) . W (K x N), all float32.
//
// An operand is taken as the sum of three bfloat16 numbers, x = h + m + l (8 + 8 + 8 bits: all 24 of it), and the product as six
// products of bfloat16 numbers, whose terms are exact: h h, h m, m h, m m, h l, l h; what is left out is below 2^-26 of a term.
// The tensor cores truncate what they add up, so a sum is theirs for 32 terms at a time only, the small products first and the
// large one last; the sums of 32 are added in registers, rounded to nearest.  Against 64 bits (2-norm of the difference over
// the result) 1.1e-7 to 1.4e-7 for sums of 1536 terms, 2.1e-7 of 4096; the library's multiply-adds on the CUDA cores are 7.0e-7
// and 1.15e-6 off.  Measured on a B200, us, library and this: 777 x 1536 x 6144 295 and 129, 777 x 1536 x 1536 104 and 41, 2048 x
// 3072 x 12352 2560 and 971 (160 TFLOP/s of 32-bit products).
//
// One persistent CTA per SM walks tiles of 128 rows x 192 columns (with split = 2 two CTAs share the sum of a tile and add
// their parts to a zeroed result; two terms have one sum, whichever comes first).  Three roles, specialised by warp:
//   warps 0-7    load 128 x 32 numbers of x and 32 x 192 of W (16-byte loads, the next step's on their way while these are
//                worked on), split them and leave three planes of each in a ring of three shared-memory stages, x K-major
//                with the 64-byte swizzle, W as it lies (N contiguous) with the 128-byte swizzle;
//   warp 16      owns the tensor memory; one lane issues the twelve products of a stage into one of two accumulators;
//   warps 8-15   add the finished accumulator to their 96 sums (a thread a row and half of the columns), and store them.
// A step takes some 2300 cycles, bound by the splitting warps (their loads' latency, the split, the look at what it loses); its products take 1152,
// shared memory (120 KB read by the products, 60 KB of planes written) 1440.  An issuing lane in one of the splitting warps
// took 1500 cycles a step of that warp's time, 3300 a step in all.  Tiles of 128 columns
// split more numbers a product; the sums of 256 columns do not fit the registers.
//
// What the split loses is computed again.  A number that is not finite does not survive it (an infinity leaves NaN), parts below
// 2^-126 of numbers below 2^-100 may be lost, however large the numbers are that they meet, and products of small numbers
// underflow part by part.  So the splitting warps keep the smallest and the largest number of a tile's operands (LowHigh), from
// which follows below which size an element of this tile may have lost a bit (Doubt: 2^-80 for ordinary operands), and
// those below it and those that are not finite are marked.  (The look costs a step 4 to 6 %: 123 and 39 us without it, of the 129 and 41.)
// When the CTA's tiles are done (nobody waits for anybody then) the summing warps compute a tile with marks once more by
// multiply-adds, 128 x 192 x 32 numbers at a time through the ring's memory, and replace the marked elements alone: another row's
// infinity does not change what a row gets.  777 x 1536 x 6144 with a row of infinities in W, which marks everything: 0.84 ms (16 ms
// with a thread walking K for each element), with one NaN in x 0.49 ms.
// All hand-offs are mbarriers; every wait is bounded and a wait that runs out sets the fault word, lets every role leave its
// loop, and the tensor memory is freed before the CTA ends.
#include "tc_common.cuh"

namespace {

using namespace tc;

constexpr int BM = 128, BN = 192, BK = 32, STAGES = 3;
constexpr int CONV = 256;                       // threads that split
constexpr int SUMS = 256;                       // threads that sum
constexpr int NTH = CONV + SUMS + 128;          // the last four warps' registers go to the others
constexpr int A_PLANE = BM * BK * 2;            // 8 KB: rows of 64 bytes
constexpr int W_BOX = BK * 64 * 2;              // 32 rows of K x 64 columns: rows of 128 bytes
constexpr int W_PLANE = BN / 64 * W_BOX;        // 12 KB
constexpr int STAGE_BYTES = 3 * (A_PLANE + W_PLANE);
constexpr int A_TASKS = BM * BK / 8 / CONV, W_TASKS = BN * BK / 8 / CONV;       // runs of eight numbers a thread
static_assert(CONV == 256 && BK == 32 && A_TASKS == 2 && W_TASKS == BN / 64, "who splits what");
constexpr int HALF = BN / 2;                    // columns of a summing thread
// A unit's LowHigh lies in one of eight places: the splitting warps are up to STAGES steps ahead of the products and these up to two of
// the sums, so they are at most six units ahead (a unit has one step or more) of what the summing warps have finished with.
constexpr int FACTS = 8;
static_assert(STAGES + 2 < FACTS, "a place is read before it is written again");
constexpr int MARK_WORDS = 32;                  // of the CTA's units (modulo 1024): those with marked elements
constexpr int X_PITCH = BK + 4;                 // multiply-adds: floats a row of x; two buffers of x and W in the ring
static_assert(2 * (BM * X_PITCH + BK * BN) <= STAGES * STAGE_BYTES / 4 && BM * BN <= STAGES * STAGE_BYTES / 4 && BM == SUMS / 2 && BN == 192,
              "who multiplies what");
constexpr unsigned ACC_COLS = 256, TMEM_COLS = 512;

struct SplitParams {
    const float *x, *w;
    float* out;
    int ldx, ldw, ldo;
    int M, N, K, tiles_m, tiles_n, split;
    int* fault;
};

// Shared-memory descriptor of a K-major operand with the 64-byte swizzle (rows of 64 bytes, eight of them a group).
__device__ __forceinline__ unsigned long long smem_desc64(unsigned addr) {
    return (unsigned long long)((addr >> 4) & 0x3FFFu) | (1ull << 16) | ((unsigned long long)(512 >> 4) << 32) | (1ull << 46) | (4ull << 61);
}

__device__ __forceinline__ void split2(float x, float y, unsigned& h, unsigned& m, unsigned& l) {
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(h) : "f"(y), "f"(x));
    x -= __uint_as_float(h << 16); y -= __uint_as_float(h & 0xffff0000u);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(m) : "f"(y), "f"(x));
    x -= __uint_as_float(m << 16); y -= __uint_as_float(m & 0xffff0000u);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(l) : "f"(y), "f"(x));
}
// eight numbers split, at the same place of three planes
__device__ __forceinline__ void store_split(unsigned char* dst, int plane_bytes, const float4& a, const float4& b) {
    uint4 h, m, l;
    split2(a.x, a.y, h.x, m.x, l.x); split2(a.z, a.w, h.y, m.y, l.y);
    split2(b.x, b.y, h.z, m.z, l.z); split2(b.z, b.w, h.w, m.w, l.w);
    *reinterpret_cast<uint4*>(dst) = h;
    *reinterpret_cast<uint4*>(dst + plane_bytes) = m;
    *reinterpret_cast<uint4*>(dst + 2 * plane_bytes) = l;
}
// four numbers, or zeros.  (In the order written: a task's next numbers are asked for as soon as its registers are free, behind the look
// at the last ones.  Left to the compiler these loads come last, and a step takes 8 % longer.)
__device__ __forceinline__ float4 load4(const float* p, bool there) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    asm volatile("{\n.reg .pred q;\nsetp.ne.b32 q, %5, 0;\n@q ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];\n}\n"
                 : "+f"(v.x), "+f"(v.y), "+f"(v.z), "+f"(v.w) : "l"(p), "r"((int)there));
    return v;
}
// 16 consecutive float32 columns of this thread's row of tensor memory
__device__ __forceinline__ void tmem_ld16(unsigned taddr, float (&v)[16]) {
    unsigned* r = reinterpret_cast<unsigned*>(v);
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                   "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr));
    tmem_ld_wait();
    tmem_ld_arrived(v);
}
// Of some operands: the smallest that is not zero and the largest, by size.  `low` is twice its bits, less one: a zero becomes the
// largest number there is.
struct LowHigh {
    unsigned low;
    float high;
    __device__ __forceinline__ void clear() { low = 0xffffffffu; high = 0.f; }
    __device__ __forceinline__ void add(float a, float b) {
        low = __vimin3_u32(low, __float_as_uint(a) * 2u - 1u, __float_as_uint(b) * 2u - 1u);
        asm("max.abs.f32 %0, %0, %1, %2;\n" : "+f"(high) : "f"(a), "f"(b));
    }
    __device__ __forceinline__ void add(const float4& v) { add(v.x, v.y); add(v.z, v.w); }
};
// Which elements of a tile are computed again: those that are not finite, and those from `from` on and below `below`.
// A part below 2^-126 that is lost from an operand below 2^-100 costs an element up to 2^-126 times the largest number on the
// other side, up to twice in each of `terms` terms: below 2^27 / 2 of that in all a bit of the element's own may be gone.  A zero is one unless
// every product of two numbers that are not zero (2^-100 at the least) shows in the sums.
struct Doubt {
    float from, below;
    __device__ __forceinline__ Doubt(unsigned low_x, unsigned low_w, float high_x, float high_w, int terms) {
        constexpr unsigned TINY = 27u << 24;                                // 2^-100, as LowHigh has it
        const bool tiny_x = low_x < TINY, tiny_w = low_w < TINY;
        const float lost = (float)terms * 0x1p-98f;
        below = 0x1p-80f;
        if (tiny_x) below = fmaxf(below, lost * high_w);
        if (tiny_w) below = fmaxf(below, lost * high_x);
        const bool zeros = tiny_x || tiny_w || (low_x >> 24) + (low_w >> 24) < 2u * 127u - 100u;
        from = zeros ? 0.f : 0x1p-149f;
    }
    __device__ __forceinline__ bool of(float v) const {
        v = fabsf(v);
        return !(v <= 3.402823466e38f) || (v < below && v >= from);
    }
};
__device__ __forceinline__ void copy16(void* dst, const float* src, bool there) {       // zeros where nothing is there
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_u32(dst)), "l"(src), "r"(there ? 16 : 0));
}

// *dst += v where v or the sum may be subnormal, which the memory's own additions of 32-bit numbers flush to zero.  Only one other CTA adds
// to an element, once.
__device__ __forceinline__ void add_in_full(float* dst, float v) {
    unsigned* word = reinterpret_cast<unsigned*>(dst);
    unsigned old = *reinterpret_cast<volatile unsigned*>(word);
    for (int i = 0; i < 4; ++i) {
        const unsigned seen = atomicCAS(word, old, __float_as_uint(__uint_as_float(old) + v));
        if (seen == old) break;
        old = seen;
    }
}

// One tile (columns k0 .. k1 of x) by multiply-adds, for the elements that are marked, by the summing threads: 16 rows a warp,
// columns 2 lane + 64 j, + 1 a lane.  `bufs`: two buffers of BM x X_PITCH numbers of x and BK x BN of W.
__device__ __forceinline__ void multiply_add(const SplitParams& p, float* bufs, int m0, int n0, int k0, int k1, const unsigned (*marks)[BN / 32]) {
    const int t = threadIdx.x - CONV, row = (t >> 5) * 16, col = (t & 31) * 2;
    constexpr int BUF = BM * X_PITCH + BK * BN;
    auto bring = [&](int k, float* xs) {
        float* ws = xs + BM * X_PITCH;
#pragma unroll 1
        for (int i = t; i < BM * BK / 4; i += SUMS) {
            const int r = i / (BK / 4), kk = i % (BK / 4) * 4;
            const bool there = m0 + r < p.M && k + kk < k1;
            copy16(xs + r * X_PITCH + kk, there ? p.x + (size_t)(m0 + r) * p.ldx + k + kk : p.x, there);
        }
#pragma unroll 1
        for (int i = t; i < BK * BN / 4; i += SUMS) {
            const int kk = i / (BN / 4), c = i % (BN / 4) * 4;
            const bool there = k + kk < k1 && n0 + c < p.N;
            copy16(ws + kk * BN + c, there ? p.w + (size_t)(k + kk) * p.ldw + n0 + c : p.w, there);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    float acc[16][6];
#pragma unroll
    for (int i = 0; i < 16; ++i)
#pragma unroll
        for (int j = 0; j < 6; ++j) acc[i][j] = 0.f;
    bring(k0, bufs);
    int b = 0;
#pragma unroll 1
    for (int k = k0; k < k1; k += BK, b ^= 1) {
        if (k + BK < k1) {
            bring(k + BK, bufs + (b ^ 1) * BUF);
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        } else
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        asm volatile("bar.sync 1, 256;\n" ::: "memory");
        const float* xs = bufs + b * BUF + row * X_PITCH;
        const float* ws = bufs + b * BUF + BM * X_PITCH + col;
#pragma unroll 1
        for (int kk = 0; kk < BK; kk += 2) {
            float2 w[2][3];
#pragma unroll
            for (int e = 0; e < 2; ++e)
#pragma unroll
                for (int j = 0; j < 3; ++j) w[e][j] = *reinterpret_cast<const float2*>(ws + (kk + e) * BN + 64 * j);
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const float2 x = *reinterpret_cast<const float2*>(xs + i * X_PITCH + kk);
#pragma unroll
                for (int e = 0; e < 2; ++e)
#pragma unroll
                    for (int j = 0; j < 3; ++j) {
                        acc[i][2 * j] = fmaf(e == 0 ? x.x : x.y, w[e][j].x, acc[i][2 * j]);
                        acc[i][2 * j + 1] = fmaf(e == 0 ? x.x : x.y, w[e][j].y, acc[i][2 * j + 1]);
                    }
            }
        }
        asm volatile("bar.sync 1, 256;\n" ::: "memory");
    }
    // through the same memory to the marked elements
#pragma unroll
    for (int i = 0; i < 16; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) *reinterpret_cast<float2*>(bufs + (row + i) * BN + col + 64 * j) = make_float2(acc[i][2 * j], acc[i][2 * j + 1]);
    asm volatile("bar.sync 1, 256;\n" ::: "memory");
#pragma unroll 1
    for (int i = t; i < BM * BN; i += SUMS) {
        const int r = i / BN, c = i % BN;
        if (m0 + r >= p.M || n0 + c >= p.N) continue;
        float* dst = p.out + (size_t)(m0 + r) * p.ldo + n0 + c;
        if (p.split > 1) {
            if (marks[r][c / 32] >> (c % 32) & 1u) add_in_full(dst, bufs[i]);
        } else if (!(*dst == *dst)) {
            *dst = bufs[i];
        }
    }
    asm volatile("bar.sync 1, 256;\n" ::: "memory");
}

__global__ void __launch_bounds__(NTH, 1) gemm_split_kernel(const SplitParams p) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* stages = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ unsigned long long full[STAGES], empty[STAGES], acc_full[2], acc_empty[2];
    __shared__ unsigned long long facts_full[FACTS];
    __shared__ uint4 facts[FACTS][CONV / 32];   // a splitting warp's LowHigh of x and W
    __shared__ unsigned marks[BM][BN / 32];     // split sums: elements of the CTA's only unit that were left out
    __shared__ unsigned marked[MARK_WORDS];
    __shared__ unsigned tmem_base_slot;
    __shared__ int abort_flag;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x;
    pdl_launch_dependents();
    if (tid == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], CONV / 32); mbar_init(&empty[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], SUMS / 32); }
        for (int i = 0; i < FACTS; ++i) mbar_init(&facts_full[i], CONV / 32);
        for (int i = 0; i < MARK_WORDS; ++i) marked[i] = 0u;
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == (CONV + SUMS) / 32) tmem_alloc(&tmem_base_slot, TMEM_COLS);
    fence_before();
    __syncthreads();
    fence_after();
    const unsigned tmem_base = tmem_base_slot;
    volatile int* abort = &abort_flag;
    const int units = p.tiles_m * p.tiles_n * p.split;
    const int steps = (p.K + BK - 1) / BK, share = (steps + p.split - 1) / p.split;
    // unit -> tile (rows first, so that the CTAs at work at a time share columns of W) and its steps of K
    auto place = [&](int unit, int& m0, int& n0, int& first, int& last) {
        const int part = unit % p.split, tile = unit / p.split;
        m0 = tile % p.tiles_m * BM;
        n0 = tile / p.tiles_m * BN;
        first = part * share;
        last = min(steps, first + share);
    };
    pdl_wait();

    // 640 threads are launched with 96 registers each: 256 x 80 + 256 x 144 + 128 x 32 are as many
    if (warp < CONV / 32) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 80;\n" ::);
        // runs of eight numbers: rows xrow, xrow + 64 of x at 8 * (tid % 4); row tid / 8 of W at 8 * (tid % 8) of every 64 columns
        const int xrow = tid >> 2, xk = (tid & 3) * 8, wk = tid >> 3, wn = (tid & 7) * 8;
        float4 xa[A_TASKS][2], wa[W_TASKS][2];
        int it = 0, round = 0;
        bool ok = true;
        for (int unit = blockIdx.x; unit < units && ok; unit += gridDim.x, ++round) {
            int m0, n0, first, last;
            place(unit, m0, n0, first, last);
            LowHigh of_x, of_w;
            of_x.clear();
            of_w.clear();
            auto fetch_x = [&](int step, int i) {
                const int k = step * BK + xk;
                const float* src = p.x + (size_t)(m0 + xrow + 64 * i) * p.ldx + k;
                const bool there = m0 + xrow + 64 * i < p.M && step < last;
                xa[i][0] = load4(src, there && k < p.K);
                xa[i][1] = load4(src + 4, there && k + 4 < p.K);
            };
            auto fetch_w = [&](int step, int i) {
                const int kw = step * BK + wk;
                const float* src = p.w + (size_t)kw * p.ldw + n0 + wn + 64 * i;
                const bool there = kw < p.K && step < last;
                wa[i][0] = load4(src, there && n0 + wn + 64 * i < p.N);
                wa[i][1] = load4(src + 4, there && n0 + wn + 64 * i + 4 < p.N);
            };
#pragma unroll
            for (int i = 0; i < A_TASKS; ++i) fetch_x(first, i);
#pragma unroll
            for (int i = 0; i < W_TASKS; ++i) fetch_w(first, i);
            for (int step = first; step < last; ++step, ++it) {
                const int s = it % STAGES;
                if (!__all_sync(0xffffffffu, mbar_wait(&empty[s], ((it / STAGES) & 1) ^ 1, abort, p.fault, 5))) { ok = false; break; }
                unsigned char* a = stages + s * STAGE_BYTES + xrow * 64 + (((tid & 3) ^ ((xrow >> 1) & 3)) << 4);
                unsigned char* w = stages + s * STAGE_BYTES + 3 * A_PLANE + wk * 128 + (((tid & 7) ^ (wk & 7)) << 4);
#pragma unroll
                for (int i = 0; i < A_TASKS; ++i) {
                    store_split(a + i * 64 * 64, A_PLANE, xa[i][0], xa[i][1]);
                    of_x.add(xa[i][0]);
                    of_x.add(xa[i][1]);
                    fetch_x(step + 1, i);
                }
#pragma unroll
                for (int i = 0; i < W_TASKS; ++i) {
                    store_split(w + i * W_BOX, W_PLANE, wa[i][0], wa[i][1]);
                    of_w.add(wa[i][0]);
                    of_w.add(wa[i][1]);
                    fetch_w(step + 1, i);
                }
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&full[s]);
            }
            if (!ok) break;
            uint4 f;
            f.x = __reduce_min_sync(0xffffffffu, of_x.low);
            f.y = __reduce_min_sync(0xffffffffu, of_w.low);
            f.z = __reduce_max_sync(0xffffffffu, __float_as_uint(of_x.high));       // (of numbers without a sign, in their order)
            f.w = __reduce_max_sync(0xffffffffu, __float_as_uint(of_w.high));
            if (lane == 0) { facts[round % FACTS][warp] = f; mbar_arrive(&facts_full[round % FACTS]); }
        }
    } else if (warp < (CONV + SUMS) / 32) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 144;\n" ::);
        const int quarter = warp & 3, half = warp >= CONV / 32 + 4 ? 1 : 0;
        const unsigned lanes = (unsigned)(quarter * 32) << 16;
        int it = 0, round = 0;
        bool ok = true;
        for (int unit = blockIdx.x; unit < units; unit += gridDim.x, ++round) {
            int m0, n0, first, last;
            place(unit, m0, n0, first, last);
            float acc[HALF];
#pragma unroll
            for (int i = 0; i < HALF; ++i) acc[i] = 0.f;
            for (int step = first; step < last; ++step, ++it) {
                const int b = it & 1;
                if (!__all_sync(0xffffffffu, mbar_wait(&acc_full[b], (it >> 1) & 1, abort, p.fault, 5))) { ok = false; break; }
                fence_after();
#pragma unroll
                for (int c = 0; c < HALF / 16; ++c) {
                    float v[16];
                    tmem_ld16(tmem_base + lanes + b * ACC_COLS + half * HALF + c * 16, v);
#pragma unroll
                    for (int i = 0; i < 16; ++i) acc[c * 16 + i] += v[i];
                }
                fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc_empty[b]);
            }
            ok = ok && __all_sync(0xffffffffu, mbar_wait(&facts_full[round % FACTS], (round / FACTS) & 1, abort, p.fault, 5));
            if (!ok) break;
            const uint4 f = facts[round % FACTS][lane % (CONV / 32)];
            const Doubt doubt(__reduce_min_sync(0xffffffffu, f.x), __reduce_min_sync(0xffffffffu, f.y),
                              __uint_as_float(__reduce_max_sync(0xffffffffu, f.z)), __uint_as_float(__reduce_max_sync(0xffffffffu, f.w)),
                              (last - first) * BK);
            const int row = m0 + quarter * 32 + lane, col0 = n0 + half * HALF;
            float* dst = p.out + (size_t)row * p.ldo + col0;
            bool any = false;
#pragma unroll
            for (int c = 0; c < HALF; c += 32) {
                unsigned again = 0u;
#pragma unroll
                for (int i = 0; i < 32; ++i)
                    if (doubt.of(acc[c + i])) {
                        again |= 1u << i;
                        acc[c + i] = p.split > 1 ? 0.f : __uint_as_float(0x7fffffffu);      // (marked by being no number)
                    }
                any = any || again != 0u;
                if (p.split > 1) marks[quarter * 32 + lane][(half * HALF + c) / 32] = again;
#pragma unroll
                for (int i = c; i < c + 32; i += 4) {
                    if (row >= p.M || col0 + i >= p.N) continue;
                    if (p.split == 1)
                        *reinterpret_cast<float4*>(dst + i) = make_float4(acc[i], acc[i + 1], acc[i + 2], acc[i + 3]);
                    else if (acc[i] != 0.f && acc[i + 1] != 0.f && acc[i + 2] != 0.f && acc[i + 3] != 0.f)
                        asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};\n" ::"l"(dst + i), "f"(acc[i]),
                                     "f"(acc[i + 1]), "f"(acc[i + 2]), "f"(acc[i + 3]) : "memory");
                    else {
                        // (adding a zero would flush what the other CTA may have left: see add_in_full)
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            if (acc[i + e] != 0.f) atomicAdd(dst + i + e, acc[i + e]);
                    }
                }
            }
            if (any) atomicOr(&marked[round / 32 % MARK_WORDS], 1u << (round % 32));
            __syncwarp();
        }
        asm volatile("bar.sync 1, 256;\n" ::: "memory");        // all marks are in place; the ring has no more reader or writer
        // (a wait that ran out in one of the warps leaves `abort` set for all of them)
        round = 0;
        for (int unit = blockIdx.x; unit < units && !*abort; unit += gridDim.x, ++round) {
            if (!(marked[round / 32 % MARK_WORDS] >> (round % 32) & 1u)) continue;
            int m0, n0, first, last;
            place(unit, m0, n0, first, last);
            multiply_add(p, reinterpret_cast<float*>(stages), m0, n0, first * BK, min(p.K, last * BK), marks);
        }
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 32;\n" ::);
        if (warp == (CONV + SUMS) / 32) {
            constexpr unsigned IDESC = instr_desc(BM, BN, true);
            const unsigned long long x0 = smem_desc64(smem_u32(stages)), w0 = smem_desc(smem_u32(stages) + 3 * A_PLANE, W_BOX, 1024);
            int it = 0;
            bool ok = true;
            for (int unit = blockIdx.x; unit < units && ok; unit += gridDim.x) {
                int m0, n0, first, last;
                place(unit, m0, n0, first, last);
                for (int step = first; step < last; ++step, ++it) {
                    const int s = it % STAGES, b = it & 1;
                    if (!__all_sync(0xffffffffu, mbar_wait_both(&acc_empty[b], ((it >> 1) & 1) ^ 1, &full[s], (it / STAGES) & 1, abort,
                                                                p.fault, 5))) { ok = false; break; }
                    fence_after();
                    if (elect_one()) {
                        // descriptors differ from the first stage's in the start address only (units of 16 bytes)
                        const unsigned long long xs = x0 + (unsigned)(s * STAGE_BYTES >> 4), ws = w0 + (unsigned)(s * STAGE_BYTES >> 4);
                        const unsigned d = tmem_base + b * ACC_COLS;
                        auto product = [&](int i, int j, bool begun) {      // planes i of x, j of W
#pragma unroll
                            for (int kk = 0; kk < BK / 16; ++kk)
                                umma(d, xs + ((i * A_PLANE + kk * 32) >> 4), ws + ((j * W_PLANE + kk * 2048) >> 4), IDESC, begun || kk > 0);
                        };
                        product(0, 2, false); product(2, 0, true); product(1, 1, true);
                        product(0, 1, true); product(1, 0, true); product(0, 0, true);
                        umma_commit(&empty[s]);
                        umma_commit(&acc_full[b]);
                    }
                    __syncwarp();
                }
            }
        }
        __syncwarp();
    }

    if (*abort) {
        // a wait ran out: products that were issued read shared memory and write tensor memory until they are done
        for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    }
    fence_before();
    __syncthreads();
    if (warp == (CONV + SUMS) / 32) {
        fence_after();
        tmem_free(tmem_base, TMEM_COLS);
    }
}

}  // namespace

// y = x . W in float32.  x (M x K, row stride ldx), W (K x N, row stride ldw), out (M x N, row stride ldo); K, N and the
// strides in elements are multiples of 4, the pointers 16-byte aligned.
TIS_API int tis_gemm_split(const void* x, int ldx, const void* w, int ldw, void* out, int ldo, int M, int N, int K, int* fault,
                           cudaStream_t stream) {
    if (M <= 0 || N <= 0) return TIS_OK;
    if (K <= 0 || (K % 4) || (N % 4) || (ldx % 4) || (ldw % 4) || (ldo % 4) || ldx < K || ldw < N || ldo < N ||
        (reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(out)) % 16) {
        tis_set_error("gemm_split: M %d N %d K %d strides %d %d %d: K, N and the strides must be multiples of 4 and the "
                      "pointers 16-byte aligned", M, N, K, ldx, ldw, ldo);
        return TIS_BAD_SIZE;
    }
    constexpr int smem = STAGES * STAGE_BYTES + 1024;
    if (cudaFuncSetAttribute(gemm_split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
        return tis_check_launch("gemm_split (shared memory)");
    SplitParams p;
    p.x = static_cast<const float*>(x); p.w = static_cast<const float*>(w); p.out = static_cast<float*>(out);
    p.ldx = ldx; p.ldw = ldw; p.ldo = ldo;
    p.M = M; p.N = N; p.K = K;
    p.tiles_m = (M + BM - 1) / BM; p.tiles_n = (N + BN - 1) / BN;
    p.fault = fault;
    // two CTAs a tile where that needs fewer rounds of steps: half of K (and a fixed cost of about four steps) each
    const int tiles = p.tiles_m * p.tiles_n, sms = sm_count(), steps = (K + BK - 1) / BK;
    const long long whole = (long long)((tiles + sms - 1) / sms) * (steps + 4);
    const long long halves = (long long)((2 * tiles + sms - 1) / sms) * ((steps + 1) / 2 + 6);
    p.split = steps >= 8 && 2 * tiles <= sms && halves < whole ? 2 : 1;    // (a CTA remembers the marks of one unit)
    if (p.split == 2 && cudaMemset2DAsync(out, (size_t)ldo * 4, 0, (size_t)N * 4, M, stream) != cudaSuccess)
        return tis_check_launch("gemm_split (memset)");
    const int units = tiles * p.split;
    tis_launch(gemm_split_kernel, dim3(units < sms ? units : sms), dim3(NTH), (size_t)smem, stream, p);
    return tis_check_launch("gemm_split");
}
