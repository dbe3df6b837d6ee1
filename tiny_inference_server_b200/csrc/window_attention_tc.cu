// Attention of long prompt portions over the paged cache on the fifth-generation tensor cores, for keys of TIS_KD and values
// of TIS_VD elements (compiled per pair of widths; the mma.sync kernel of window_attention_mma.cu takes all else):
//   score = q . k * scale (bounded by a tanh if asked) - r1[head] * ln(1 + r2[head] * distance), keys first_key(pos, window) ..
//   pos (common.cuh), softmax in 32-bit, out = softmax . v * sigmoid(gate).
// The roles, rings and hand-offs are those of attention_tc.cu; what differs:
//   * keys and values have widths of their own; their rows lie in the pages as they are, so the TMA engine swizzles the boxes;
//   * the value rows may be the first TIS_VD elements of the key rows (SHARED): the key tile is then read a second time as the
//     values, there is no ring of values and a slot is free when the tile's second product is done;
//   * the bias costs a logarithm an element;
//   * rows of the value tile that no row of queries sees (before the window, behind the last row, pages of others) are zeroed:
//     a probability of 0 must not meet what another request left there.
// Bound by the chain of a tile through scores, softmax and second product (two tiles side by side), as attention_tc.cu.
// Against the mma.sync kernel, which reads every operand fragment from shared memory per warp of 16 rows: 2048 rows, 12 query
// heads of 128 on 3 kv heads, window 1024, with bias 103 -> 33 us; 1024 rows behind 1024 cached, 12 heads on one
// compressed row of 192 (values 128) 201 -> 39 us (replayed from a graph); outputs against 64 bits 0.97 to 1.0 times as far off.
// With a gate the division a/(1 + e^-g) was 13000 of a tile's last cycles, an element after the other: same rows with bias and gate
// 44 us, with rows stored from shared memory and quotient() 37.
#include "tc_common.cuh"

#ifndef TIS_KD
#define TIS_KD 128
#endif
#ifndef TIS_VD
#define TIS_VD 128
#endif

// shared memory: queries, two P buffers, and two slots of keys and of values, or of both in one
#define TIS_WTC_SEPARATE (256 * TIS_KD + 65536 + 512 * (TIS_KD + TIS_VD) + 1024 <= 230400)
#define TIS_WTC_SHARED (TIS_KD >= TIS_VD && 256 * TIS_KD + 65536 + 512 * TIS_KD + 1024 <= 230400)
#if (TIS_KD % 64 == 0) && (TIS_VD % 64 == 0) && (TIS_VD <= 128) && (TIS_WTC_SEPARATE || TIS_WTC_SHARED)

namespace {

using namespace tc;

constexpr int KD = TIS_KD, VD = TIS_VD;
constexpr int K_BLOCKS = KD / 64, V_BLOCKS = VD / 64;       // 128-byte column blocks of a row
constexpr int BM = 128;                     // query rows of a CTA
constexpr int BN = 128;                     // keys of a tile
constexpr int NTH = 512;
constexpr int HALF_BYTES = 128 * 128;       // 128 rows x 128 bytes: one swizzled column block
constexpr int Q_BYTES = K_BLOCKS * HALF_BYTES;
constexpr int P_BYTES = 2 * HALF_BYTES;     // 128 rows x 128 keys, bfloat16 (one per softmax group)
constexpr int K_BYTES = K_BLOCKS * HALF_BYTES, V_BYTES = V_BLOCKS * HALF_BYTES;      // keys, values of one tile
constexpr int SLOTS = 2;                    // per ring
constexpr int PAGES_AHEAD = 3;
constexpr unsigned TMEM_COLS = 512;
constexpr unsigned COL_S = 0;               // two score buffers of 128 columns
constexpr unsigned COL_O = 256;             // two output accumulators of up to 128 columns

struct WtcParams {
    bf16* out; int out_stride;
    const int* block_table; int bt_stride; int num_pages;
    const int* positions; const int* row_slot;
    const int* tile_row0; const int* tile_rows; int num_tiles;
    int H, G, page_size, window;
    float scale_log2;
    SoftCap cap;            // bounds the raw scores (k 0: not)
    const float *r1, *r2;   // per query head (r1 null: no bias)
    const bf16* gate; int ldg, gate_per_head;       // (n, H * VD) or, per head, (n, H) (null: none)
    const float* sink;      // per query head: exp(sink) is one more term of the softmax's denominator (null: none)
    int* fault;
};

__device__ __forceinline__ float fast_log2(float x) {
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
    return y;
}
// Rows of a tile (`blocks` column blocks of 128 rows) that lie outside first .. end - 1: zeros.  By a whole warp.
__device__ __forceinline__ void zero_rows(unsigned char* tile, int blocks, int first, int end, int lane) {
    if (first <= 0 && end >= 128) return;
    for (int i = lane; i < 128 * 8 * blocks; i += 32) {
        const int row = i / 8 % 128;
        if (row < first || row >= end)
            *reinterpret_cast<uint4*>(tile + i / 1024 * HALF_BYTES + row * 128 + i % 8 * 16) = make_uint4(0u, 0u, 0u, 0u);
    }
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    __syncwarp();
}

__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
    return y;
}

// BIAS: scores have a bias (and are not bounded); SHARED: the values are the first VD elements of the key rows.
template <bool BIAS, bool SHARED>
__global__ void __launch_bounds__(NTH, 1)
window_attention_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                           const __grid_constant__ CUtensorMap map_v, const WtcParams p) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char* q_smem = base;
    unsigned char* p_smem = base + Q_BYTES;
    unsigned char* k_slots = p_smem + 2 * P_BYTES;
    unsigned char* v_slots = SHARED ? k_slots : k_slots + SLOTS * K_BYTES;
    __shared__ unsigned long long q_full, full_k[SLOTS], empty_k[SLOTS], full_v[SLOTS], empty_v[SLOTS], s_full[2], s_free[2], p_full[2], o_done[2], turn[2];
    __shared__ unsigned tmem_base_slot;
    __shared__ int abort_flag;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    pdl_launch_dependents();

    // heaviest tiles (the last rows of a prompt see the most keys) first
    const int tile = p.num_tiles - 1 - (int)blockIdx.x / p.H;
    const int head = (int)blockIdx.x % p.H;
    const int kvh = head / (p.H / p.G);
    const int row0 = p.tile_row0[tile];
    const int nrows = min(p.tile_rows[tile], BM);
    if (nrows <= 0) return;
    // A stage that runs behind the trunk sees the first rows of a prompt as padding (slot -1,
    // position 0): the tile's request and last position are those of its last row.
    const int slot = p.row_slot[row0 + nrows - 1];
    if (slot < 0) return;                                 // padding only: the whole CTA leaves together
    const int pos0 = p.positions[row0];                   // the smallest position of the tile
    const int hi = p.positions[row0 + nrows - 1] + 1;     // keys [.., hi) are visible to the last row
    const int lo_first = first_key(pos0, p.window);
    const int tile_begin = lo_first & ~(BN - 1);
    const int T = (hi - tile_begin + BN - 1) / BN;

    if (threadIdx.x == 0) {
        mbar_init(&q_full, 1);
        for (int s = 0; s < SLOTS; ++s) {
            mbar_init(&full_k[s], SHARED ? 4 : 2); mbar_init(&empty_k[s], 1);
            mbar_init(&full_v[s], 2); mbar_init(&empty_v[s], 1);
        }
        mbar_init(&s_full[0], 1); mbar_init(&s_full[1], 1);
        mbar_init(&s_free[0], 4); mbar_init(&s_free[1], 4);
        mbar_init(&p_full[0], 4); mbar_init(&p_full[1], 4);
        mbar_init(&turn[0], 4); mbar_init(&turn[1], 4);
        mbar_init(&o_done[0], 1); mbar_init(&o_done[1], 1);
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        prefetch_map(&map_q);
        prefetch_map(&map_k);
        if (!SHARED) prefetch_map(&map_v);
    }
    if (warp == 1) tmem_alloc(&tmem_base_slot, TMEM_COLS);
    fence_before();
    __syncthreads();
    fence_after();
    const unsigned tmem_base = tmem_base_slot;
    volatile int* abort = &abort_flag;
    pdl_wait();                                           // q and the cache rows of this step come from the kernel before

    // 512 threads are launched with 128 registers each, 65536 in all: 256 x 40 + 256 x 216
    if (warp < 4 || warp >= 12) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 40;\n" ::);
        if (warp == 0 || warp == 2 || warp == 12 || warp == 13) {
            // ---- loads: warps 0 and 12 keys (and Q), warps 2 and 13 values, or keys as well --------------
            const int kv = SHARED || warp == 0 || warp == 12 ? 0 : 1, parts = SHARED ? 4 : 2;
            const int part = (warp >= 12 ? 1 : 0) + (SHARED && (warp == 2 || warp == 13) ? 2 : 0);
            unsigned long long* full = kv ? full_v : full_k;
            unsigned long long* empty = kv ? empty_v : empty_k;
            unsigned char* ring = kv ? v_slots : k_slots;
            const int blocks = kv ? V_BLOCKS : K_BLOCKS, boxes = BN / p.page_size * blocks;    // boxes of a key tile (1..32)
            const bool mine = lane < boxes && lane % parts == part;           // a lane a box, the warps taking turns
            const int part_bytes = (boxes + parts - 1 - part) / parts * p.page_size * 128, in_tile = lane / blocks * p.page_size;
            const int* bt = p.block_table + (size_t)slot * p.bt_stride;
            // (as in attention_tc.cu: read PAGES_AHEAD tiles before they are looked at)
            auto page_of = [&](int j) -> int {
                const int key0 = tile_begin + j * BN + in_tile;
                if (j >= T || !mine || key0 >= hi || key0 + p.page_size <= lo_first) return 0;  // no row sees it: any page will do
                return bt[key0 / p.page_size];
            };
            if (warp == 0 && lane == 0) {
                mbar_arrive_expect_tx(&q_full, Q_BYTES);
#pragma unroll
                for (int hh = 0; hh < K_BLOCKS; ++hh)
                    tma_load_2d(q_smem + hh * HALF_BYTES, &map_q, head * KD + hh * 64, row0, &q_full);
            }
            int pages[PAGES_AHEAD];
#pragma unroll
            for (int a = 0; a < PAGES_AHEAD; ++a) pages[a] = page_of(a);
            for (int j = 0; j < T; ++j) {
                int page = pages[0];
#pragma unroll
                for (int a = 1; a < PAGES_AHEAD; ++a) pages[a - 1] = pages[a];
                pages[PAGES_AHEAD - 1] = page_of(j + PAGES_AHEAD);
                const int s = j % SLOTS;
                if (!__all_sync(0xffffffffu, mbar_wait(&empty[s], ((j / SLOTS) & 1) ^ 1, abort, p.fault, 6))) break;
                if (page < 0 || page >= p.num_pages) { atomicExch(p.fault, 5); page = 0; }
                if (lane == 0) mbar_arrive_expect_tx(&full[s], part_bytes);
                __syncwarp();
                if (mine) {
                    const int block = lane % blocks;
                    tma_load_3d(ring + (size_t)s * (kv ? V_BYTES : K_BYTES) + block * HALF_BYTES + in_tile * 128, kv ? &map_v : &map_k,
                                block * 64, kvh * p.page_size, page, &full[s]);
                }
            }
        } else if (warp == 1) {
            // ---- products, first kind: S_j = Q K_j^T into score buffer j & 1 ----------------------------
            constexpr unsigned IDESC_S = instr_desc(BM, BN, false);
            const unsigned long long q_desc0 = smem_desc(smem_u32(q_smem), 16, 1024);
            const unsigned long long k_desc0 = smem_desc(smem_u32(k_slots), 16, 1024);
            bool ok = mbar_wait(&q_full, 0, abort, p.fault, 6);
            for (int j = 0; j < T; ++j) {
                const int g = j & 1, i = j >> 1, s = j % SLOTS;
                // the group has the scores of its tile before in registers
                ok = ok && (i == 0 ? mbar_wait(&full_k[s], (j / SLOTS) & 1, abort, p.fault, 6)
                                   : mbar_wait_both(&s_free[g], (i - 1) & 1, &full_k[s], (j / SLOTS) & 1, abort, p.fault, 6));
                if (!__all_sync(0xffffffffu, ok)) break;
                if (SHARED && (j == 0 || j == T - 1))
                    zero_rows(k_slots + s * K_BYTES, V_BLOCKS, lo_first - (tile_begin + j * BN), hi - (tile_begin + j * BN), lane);
                fence_after();
                if (elect_one()) {
                    // descriptors differ from the ring's first one only in the start address (units of 16 bytes)
                    const unsigned long long kd = k_desc0 + (unsigned long long)((s * K_BYTES) >> 4);
                    const unsigned d = tmem_base + COL_S + g * BN;
#pragma unroll
                    for (int kk = 0; kk < KD / 16; ++kk) {
                        const unsigned long long off = (unsigned long long)(((kk >> 2) * HALF_BYTES + (kk & 3) * 32) >> 4);
                        umma(d, q_desc0 + off, kd + off, IDESC_S, kk != 0);
                    }
                    if (!SHARED) umma_commit(&empty_k[s]);
                    umma_commit(&s_full[g]);
                }
                __syncwarp();
            }
        } else if (warp == 3) {
            // ---- products, second kind: O_g += P_j V_j.  An issuing warp of its own: while one waits for a barrier the
            // other keeps the tensor cores fed. --------------------------------------------------------------
            constexpr unsigned IDESC_O = instr_desc(BM, VD, true);
            constexpr int SLOT = SHARED ? K_BYTES : V_BYTES;
            const unsigned long long p_desc0 = smem_desc(smem_u32(p_smem), 16, 1024);
            const unsigned long long v_desc0 = smem_desc(smem_u32(v_slots), HALF_BYTES, 1024);
            for (int j = 0; j < T; ++j) {
                const int g = j & 1, i = j >> 1, s = j % SLOTS;
                bool ok = SHARED || mbar_wait(&full_v[s], (j / SLOTS) & 1, abort, p.fault, 6);
                if (!__all_sync(0xffffffffu, ok)) break;
                if (!SHARED && (j == 0 || j == T - 1))
                    zero_rows(v_slots + s * V_BYTES, V_BLOCKS, lo_first - (tile_begin + j * BN), hi - (tile_begin + j * BN), lane);
                ok = mbar_wait(&p_full[g], i & 1, abort, p.fault, 6);
                if (!__all_sync(0xffffffffu, ok)) break;
                fence_after();
                if (elect_one()) {
                    const unsigned long long vd = v_desc0 + (unsigned long long)((s * SLOT) >> 4);
                    const unsigned long long pd = p_desc0 + (unsigned long long)((g * P_BYTES) >> 4);
                    const unsigned d = tmem_base + COL_O + g * 128;
#pragma unroll
                    for (int kk = 0; kk < BN / 16; ++kk) {    // 16 keys: 32 bytes along a row of P, 16 rows of V
                        umma(d, pd + (unsigned long long)(((kk >> 2) * HALF_BYTES + (kk & 3) * 32) >> 4),
                             vd + (unsigned long long)((kk * 2048) >> 4), IDESC_O, (i | kk) != 0);
                    }
                    umma_commit(SHARED ? &empty_k[s] : &empty_v[s]);
                    umma_commit(&o_done[g]);
                }
                __syncwarp();
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 216;\n" ::);
        // ---- softmax: one thread per query row in each of the two groups ----------------------
        const int g = warp >= 8 ? 1 : 0;                  // warps 4-7 and 8-11
        const int quarter = warp & 3;                     // the lanes of tensor memory this warp may touch
        const int r = quarter * 32 + lane;
        const bool row_ok = r < nrows && p.row_slot[row0 + r] >= 0;
        const int qpos = row_ok ? p.positions[row0 + r] : 0;
        const int lo_r = first_key(qpos, p.window);
        const int lo_last = first_key(hi - 1, p.window);                   // the last row's first key
        const float b1 = BIAS ? p.r1[head] : 0.f, b2 = BIAS ? p.r2[head] : 0.f;
        const unsigned lane_bits = (unsigned)(quarter * 32) << 16;
        const unsigned col_s = COL_S + g * BN, col_o = COL_O + g * 128;
        unsigned char* pg_smem = p_smem + g * P_BYTES;
        const bool warp_has_rows = __any_sync(0xffffffffu, row_ok);
        float m_used = -INFINITY, l_sum = 0.f;
        bool ok = true;
        // before the exponentials of the group's tile i: the products of its tile before are done, and the other group's
        // exponentials of the tile before in the row's order.  (Left to themselves the groups come to their exponentials
        // together and share the units: each 2000 cycles for what takes one alone 1100.)
        auto wait_turn = [&](int i) {
            if (g == 0) return i == 0 || mbar_wait_both(&o_done[0], (i - 1) & 1, &turn[0], (i - 1) & 1, abort, p.fault, 6);
            return i == 0 ? mbar_wait(&turn[1], 0, abort, p.fault, 6)
                          : mbar_wait_both(&o_done[1], (i - 1) & 1, &turn[1], i & 1, abort, p.fault, 6);
        };
        int i = 0;                                        // tiles of this group so far
        for (int j = g; j < T; j += 2, ++i) {
            if (!__all_sync(0xffffffffu, mbar_wait(&s_full[g], i & 1, abort, p.fault, 6))) { ok = false; break; }
            fence_after();
            if (!warp_has_rows) {
                // a warp whose 32 rows are all beyond the tile: its rows of P are zero, once and for all
                if (i == 0) {
#pragma unroll
                    for (int c = 0; c < 16; ++c)
                        *reinterpret_cast<uint4*>(pg_smem + r * 128 + (c >> 3) * HALF_BYTES + ((c & 7) << 4)) = make_uint4(0u, 0u, 0u, 0u);
                    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                }
                // it follows every phase of o_done and turn all the same: a wait for the last one alone could return a phase
                // early (the parity of the phase before the one before), and the merge below writes where P lies
                if (!__all_sync(0xffffffffu, wait_turn(i))) { ok = false; break; }
                if (lane == 0) mbar_arrive(&turn[1 - g]);
                fence_before();
                __syncwarp();
                if (lane == 0) { mbar_arrive(&s_free[g]); mbar_arrive(&p_full[g]); }
                continue;
            }
            const int kt = tile_begin + j * BN;
            const bool whole = kt + BN - 1 <= pos0 && kt >= lo_last;      // every row of the tile sees every key
            float s[BN];
#pragma unroll
            for (int c = 0; c < BN / 32; ++c) tmem_ld32_issue(tmem_base + lane_bits + col_s + c * 32, s + c * 32);
            tmem_ld_wait();
            tmem_ld_arrived(s);
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&s_free[g]);
            // with a bias: in units of log2 from here on; without, the scale is left to the exponentials
            if (BIAS) {
                const float d0 = (float)(qpos - kt);
#pragma unroll
                for (int e = 0; e < BN; ++e) s[e] = fmaf(s[e], p.scale_log2, -b1 * fast_log2(fmaf(b2, d0 - (float)e, 1.f)));
            } else if (p.cap.k != 0.f) {
#pragma unroll
                for (int e = 0; e < BN; ++e) s[e] = soft_capped(s[e], p.cap);
            }
            if (!(whole && row_ok)) {
                // keys lo_r .. qpos, counted from the tile's first; a padding row sees none
                const int from = row_ok ? lo_r - kt : 1 << 20, span = row_ok ? qpos - lo_r : 0;
#pragma unroll
                for (int e = 0; e < BN; ++e) s[e] = (unsigned)(e - from) <= (unsigned)span ? s[e] : -INFINITY;
            }
            // the row's maximum (the scale is positive)
            float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int e = 0; e < BN; ++e) mx4[e & 3] = fmaxf(mx4[e & 3], s[e]);
            float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
            if (!BIAS) mx *= p.scale_log2;
            // the reference is the row's maximum itself, so that the largest probability is 1 and not rounded.  (Raised only
            // when the maximum had left it far behind: 1 to 2 % more error of the outputs, 2 % less time.)
            const bool raise = mx > m_used;
            float alpha = 1.f;
            if (raise) {
                alpha = m_used == -INFINITY ? 0.f : fast_exp2(m_used - mx);
                m_used = mx;
                l_sum *= alpha;
            }
            // the products of the group's tile before are done: O may be rescaled, P overwritten
            if (!__all_sync(0xffffffffu, wait_turn(i))) { ok = false; break; }
            if (i > 0 && __any_sync(0xffffffffu, raise)) {
                fence_after();
#pragma unroll 1
                for (int c = 0; c < VD / 64; ++c) {
                    float o[2][32];
                    const unsigned at = tmem_base + lane_bits + col_o + c * 64;
                    tmem_ld32_issue(at, o[0]);
                    tmem_ld32_issue(at + 32, o[1]);
                    tmem_ld_wait();
                    tmem_ld_arrived(o[0]);
                    tmem_ld_arrived(o[1]);
#pragma unroll
                    for (int e = 0; e < 64; ++e) o[e >> 5][e & 31] *= alpha;
                    tmem_st32(at, o[0]);
                    tmem_st32(at + 32, o[1]);
                }
                fence_before();
            }
            const float neg_m = m_used == -INFINITY ? 0.f : -m_used;
            float ps4[4] = {0.f, 0.f, 0.f, 0.f};
            unsigned char* prow = pg_smem + r * 128;
            const float sc = BIAS ? 1.f : p.scale_log2;
#pragma unroll
            for (int c = 0; c < BN / 8; ++c) {            // eight keys: one 16-byte chunk of the row of P
                unsigned pk[4];
#pragma unroll
                for (int e = 0; e < 8; e += 2) {
                    const float a = fast_exp2(fmaf(s[c * 8 + e], sc, neg_m));                 // 2^-inf = 0 for masked keys
                    const float b = fast_exp2(fmaf(s[c * 8 + e + 1], sc, neg_m));
                    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
                    pk[e >> 1] = *reinterpret_cast<unsigned*>(&h);
                    // the sum of what the product sees: a row that is nearly all one key's comes out as that key's value
                    ps4[e >> 1] += __uint_as_float(pk[e >> 1] << 16) + __uint_as_float(pk[e >> 1] & 0xffff0000u);
                }
                *reinterpret_cast<uint4*>(prow + (c >> 3) * HALF_BYTES + (((c & 7) ^ (r & 7)) << 4)) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
                if (c == BN / 16 - 1 && lane == 0) mbar_arrive(&turn[1 - g]);
            }
            l_sum += (ps4[0] + ps4[1]) + (ps4[2] + ps4[3]);
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_full[g]);
        }
        // ---- merge the two groups' halves, each group half of the columns, and store them through the ring of keys, which
        // has no more copies or products to come once both groups' last products are done --------------------------
        typedef StagedRows<VD> Rows;
        float* stage = reinterpret_cast<float*>(k_slots);
        const int first = Rows::row(warp - 4, lane, 0), col = Rows::col(lane);
        bf16* dst = p.out + (size_t)(row0 + first) * p.out_stride + head * VD + col;
        const bool gated = p.gate != nullptr && !p.gate_per_head;
        uint2 gates[4];                                   // of the next four steps, on their way
        auto fetch_gates = [&](int i0) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int at = first + (i0 + i) * Rows::ROWS;
                gates[i] = make_uint2(0u, 0u);
                if (gated && at < nrows) gates[i] = *reinterpret_cast<const uint2*>(p.gate + (size_t)(row0 + at) * p.ldg + (size_t)head * VD + col);
            }
        };
        fetch_gates(0);
        if (i > 0 && ok) ok = __all_sync(0xffffffffu, mbar_wait(&o_done[g], (i - 1) & 1, abort, p.fault, 6));
        // the group's P buffer is free now: it carries the row's maximum and sum to the other group
        reinterpret_cast<float*>(pg_smem)[r] = m_used;
        reinterpret_cast<float*>(pg_smem)[BM + r] = l_sum;
        fence_before();
        asm volatile("bar.sync 1, 256;\n" ::: "memory");        // both groups' products are done, sums are in place
        fence_after();
        if (ok && !*abort) {
            const float* mg0 = reinterpret_cast<const float*>(p_smem);
            const float* mg1 = reinterpret_cast<const float*>(p_smem + P_BYTES);
            const float m0 = mg0[r], m1 = mg1[r], l0 = mg0[BM + r], l1 = mg1[BM + r];
            const float sink2 = p.sink != nullptr ? p.sink[head] * 1.4426950408889634f : -INFINITY;
            const float m = fmaxf(fmaxf(m0, m1), sink2);
            const float w0 = m0 == -INFINITY ? 0.f : fast_exp2(m0 - m);
            const float w1 = (T < 2 || m1 == -INFINITY) ? 0.f : fast_exp2(m1 - m);
            const float l = l0 * w0 + l1 * w1 + (sink2 == -INFINITY ? 0.f : fast_exp2(sink2 - m));
            float inv = l > 0.f ? 1.f / l : 0.f;
            if (p.gate != nullptr && p.gate_per_head && r < nrows) inv /= 1.f + __expf(-__bfloat162float(p.gate[(size_t)(row0 + r) * p.ldg + head]));
            constexpr int COLS = VD / 2;                  // this group's share of the columns
#pragma unroll
            for (int c = 0; c < COLS / 32; ++c) {
                const int col = g * COLS + c * 32;
                float o0[32], o1[32];
                tmem_ld32_issue(tmem_base + lane_bits + COL_O + col, o0);
                if (T >= 2) tmem_ld32_issue(tmem_base + lane_bits + COL_O + 128 + col, o1);
                tmem_ld_wait();
                tmem_ld_arrived(o0);
                if (T >= 2) tmem_ld_arrived(o1);
                // padding rows inside the tile get zeros
#pragma unroll
                for (int e = 0; e < 32; ++e) o0[e] = row_ok ? (o0[e] * w0 + (T >= 2 ? o1[e] * w1 : 0.f)) * inv : 0.f;
                stage_put<VD>(stage, r, col, o0);
            }
            fence_before();
        }
        asm volatile("bar.sync 1, 256;\n" ::: "memory");
        if (!*abort) {
#pragma unroll 1                                          // (code that runs once takes longer to fetch than to run)
            for (int i0 = 0; i0 < Rows::STEPS; i0 += 4, dst += (size_t)4 * Rows::ROWS * p.out_stride) {
                uint2 now[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) now[i] = gates[i];
                if (i0 + 4 < Rows::STEPS) fetch_gates(i0 + 4);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int at = first + (i0 + i) * Rows::ROWS;
                    float4 v = Rows::get(stage, at, col);
                    if (gated) {
                        v.x = quotient(v.x, 1.f + __expf(-__uint_as_float(now[i].x << 16)));
                        v.y = quotient(v.y, 1.f + __expf(-__uint_as_float(now[i].x & 0xffff0000u)));
                        v.z = quotient(v.z, 1.f + __expf(-__uint_as_float(now[i].y << 16)));
                        v.w = quotient(v.w, 1.f + __expf(-__uint_as_float(now[i].y & 0xffff0000u)));
                    }
                    if (at < nrows) store4(dst + (size_t)i * Rows::ROWS * p.out_stride, v);
                }
            }
        }
    }

    if (*abort) {
        // a wait ran out: give copies that may still be in flight time to land before the
        // shared memory is given up
        for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    }
    fence_before();
    __syncthreads();
    if (warp == 1) {
        fence_after();
        tmem_free(tmem_base, TMEM_COLS);
    }
}

template <bool BIAS, bool SHARED>
int launch_wtc(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const WtcParams& p, cudaStream_t stream) {
    constexpr int smem = Q_BYTES + 2 * P_BYTES + SLOTS * (K_BYTES + (SHARED ? 0 : V_BYTES)) + 1024;
    if (cudaFuncSetAttribute(window_attention_tc_kernel<BIAS, SHARED>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
        return tis_check_launch("window_attention_tc (shared memory)");
    tis_launch(window_attention_tc_kernel<BIAS, SHARED>, dim3(p.num_tiles * p.H), dim3(NTH), (size_t)smem, stream, mq, mk, mv, p);
    return tis_check_launch("window_attention_tc");
}

}  // namespace

// Which forms this pair of widths has: 1 values of their own, 2 values that are the first elements of the key rows, 3 both.
TIS_API int tis_window_attention_tc_forms() { return (TIS_WTC_SEPARATE ? 1 : 0) | (TIS_WTC_SHARED ? 2 : 0); }

// Attention of `num_tiles` tiles of up to 128 consecutive rows of one request each.  q is (n, >= H * KD) with row stride ldq,
// out (n, H * VD); a page's key rows [G, page_size, KD] lie side by side, its value rows [G, page_size, VD] likewise, or
// (`shared`) they are the first VD elements of the key rows; page_size 16, 32, 64 or 128.  scale > 0.  Rows of q, out, the
// pages and an element-by-element gate start on 16-byte boundaries (strides multiples of 8).
TIS_API int tis_window_attention_tc(const void* q, int ldq, int n_rows, const void* gate, int ldg, int gate_per_head, void* out,
                                    int ldo, const void* k_pages, size_t k_page_stride, const void* v_pages,
                                    size_t v_page_stride, int shared, const int* block_table, int bt_stride, int num_pages,
                                    const int* positions, const int* row_slot, const int* tile_row0, const int* tile_rows,
                                    int num_tiles, int H, int G, int page_size, int window, float scale, float softcap,
                                    const float* r1, const float* r2, const float* sink, int* fault, cudaStream_t stream) {
    if (num_tiles <= 0) return TIS_OK;
    const bool elementwise = gate != nullptr && !gate_per_head;
    if ((page_size != 16 && page_size != 32 && page_size != 64 && page_size != 128) || H <= 0 || G <= 0 || H % G || !(scale > 0.f) ||
        ldq % 8 || ldo % 8 || k_page_stride % 8 || v_page_stride % 8 || (elementwise && ldg % 8) ||
        ((uintptr_t)q | (uintptr_t)out | (uintptr_t)k_pages | (uintptr_t)v_pages | (elementwise ? (uintptr_t)gate : (uintptr_t)0)) % 16 ||
        (r1 != nullptr && (softcap > 0.f || window < 0)) || !((tis_window_attention_tc_forms() >> (shared ? 1 : 0)) & 1) ||
        (long long)num_tiles * H > 0x7fffffff) {
        tis_set_error("window_attention_tc: %d query heads on %d, page size %d, scale %g, strides %d/%d/%d, values %s, or operands "
                      "that are not aligned", H, G, page_size, scale, ldq, ldg, ldo, shared ? "in the key rows" : "of their own");
        return TIS_BAD_SIZE;
    }
    CUtensorMap mq, mk, mv;
    if (!tensor_map(q, (long long)H * KD, n_rows, ldq, BM, true, &mq)) return TIS_CUDA_ERROR;
    if (!page_map(k_pages, KD, G * page_size, num_pages, KD, k_page_stride, page_size, &mk)) return TIS_CUDA_ERROR;
    if (shared) mv = mk;
    else if (!page_map(v_pages, VD, G * page_size, num_pages, VD, v_page_stride, page_size, &mv)) return TIS_CUDA_ERROR;
    WtcParams p;
    p.out = static_cast<bf16*>(out); p.out_stride = ldo;
    p.block_table = block_table; p.bt_stride = bt_stride; p.num_pages = num_pages;
    p.positions = positions; p.row_slot = row_slot;
    p.tile_row0 = tile_row0; p.tile_rows = tile_rows; p.num_tiles = num_tiles;
    p.H = H; p.G = G; p.page_size = page_size; p.window = window;
    p.scale_log2 = scale * 1.4426950408889634f;
    p.cap = soft_cap(softcap, scale);
    p.r1 = r1; p.r2 = r2;
    p.gate = static_cast<const bf16*>(gate); p.ldg = ldg; p.gate_per_head = gate_per_head;
    p.sink = sink;
    p.fault = fault;
#if TIS_WTC_SHARED
    if (shared) return r1 != nullptr ? launch_wtc<true, true>(mq, mk, mv, p, stream) : launch_wtc<false, true>(mq, mk, mv, p, stream);
#endif
#if TIS_WTC_SEPARATE
    return r1 != nullptr ? launch_wtc<true, false>(mq, mk, mv, p, stream) : launch_wtc<false, false>(mq, mk, mv, p, stream);
#else
    return TIS_BAD_SIZE;
#endif
}

#else

TIS_API int tis_window_attention_tc_forms() { return 0; }

TIS_API int tis_window_attention_tc(const void*, int, int, const void*, int, int, void*, int, const void*, size_t, const void*,
                                    size_t, int, const int*, int, int, const int*, const int*, const int*, const int*, int, int,
                                    int, int, int, float, float, const float*, const float*, const float*, int*, cudaStream_t) {
    tis_set_error("window_attention_tc: built for widths it does not take");
    return TIS_BAD_SIZE;
}

#endif
