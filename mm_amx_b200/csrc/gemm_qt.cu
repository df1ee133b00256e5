// Fully-connected layer with int8-compressed or 4-bit weights and more than 16 rows of bf16 activations.
//
// Replaces the M > 16 branches of the compressed-weight specialisation Matmul<bf16,int8_t,float> (include/kernels_amx.hpp:1443-1514),
// which decompresses 16 weight rows at a time in front of the tile product.  Here the weights cross HBM, L2 and shared memory as they are
// stored, are widened to bf16 in registers and go from there into tensor memory, one weight row per lane, as the A operand of
// tcgen05.mma; the activations are the B operand, as TMA brings them.  The product is therefore the transposed one:
// D [weight rows x tokens] = W [weight rows x K] * X^T.  Widened weights in shared memory would cost it two more passes (the
// store and the MMA's operand read), which is more than its bandwidth beside the activations, and widened weights in global memory a
// second trip through L2.
//
// A CTA, or a pair of CTAs (cta_group::2, each with 128 weight rows and half of the tokens' loads), walks tiles of 128 / 256 weight
// rows x T tokens; with few tiles S CTAs or pairs share the K of a tile and meet in distributed shared memory.  An accumulator is
// drained by warps of its own while the next tile multiplies.
//   int8   : exact in bf16; scales in the epilogue.   4 bits : value x group scale in fp32, rounded once to bf16.
// Where K must be summed in several chains (the tensor core's error grows with a chain's length) its parts go to one accumulator
// after the other, and the epilogue warps add them in registers (FOLD).
//
// Warps: 0 = TMA loads of activations, 1 = MMA issue and TMEM owner, 2 = TMA loads of weights, 3 idle, 4-11 = epilogue (two per TMEM
// quarter), 12-19 = widening in two sets of four (one warp per TMEM quarter) that take the pieces of 128 rows x 128 K in turn.
// Barriers: x_full (in the pair's leader) / x_empty per slot of activations, raw_full / raw_empty per slot of stored weights, a_full (in
// the leader) / a_empty per A buffer in tensor memory, d_full / d_empty (in the leader) per accumulator.  Every wait is bounded as in gemm_tc.cu.
#include <cmath>
#include "split_k.h"
#include "tc_common.cuh"

namespace b200fc {

namespace {

constexpr int QT_ROWS = 128;                          // weight rows per CTA
constexpr int PIECE_K = 128;                          // K of a piece: an A buffer of 64 columns of tensor memory
constexpr int A_COLS = 64;
// (Two sets of each: 640 threads, 96 registers.  One set of epilogue warps: int8 1071 x 2560 x 22784 with GeLU 147 us instead of 116.)
constexpr int QT_SETS = 2, QT_EPI_SETS = 2, QT_EPI_WARPS = 4 * QT_EPI_SETS;
static_assert(QT_SETS == 2, "see run_qt on the slots");
constexpr int QT_THREADS = 128 * (1 + QT_EPI_SETS + QT_SETS);
constexpr int FIRST_WIDENER = 4 + QT_EPI_WARPS;
constexpr int MAX_X = 16, MAX_RAW = 6, MAX_A = 6, MAX_D = 8;
constexpr int QT_BAR_BYTES = 768;
constexpr int QT_SMEM = 232448;                       // all an SM gives to one CTA
constexpr int QT_RING = (QT_SMEM - 1024 - QT_BAR_BYTES) / 1024 * 1024;
constexpr int RAW_BYTES = QT_ROWS * SLAB_BYTES;       // a stored piece: 128 rows x 128 bytes
constexpr int CHUNK = 16;                             // tokens that an epilogue warp takes at a time
constexpr int CHUNK_BYTES = CHUNK * QT_ROWS * 4;      // their partial sums

struct QtParams {
    int M, n0, n1, row_blocks;     // row_blocks: of the packed matrix (128 rows each)
    int T, tiles_m, tiles_n, S, parts;
    int stages;                    // stored pieces per weight row
    int x_slots, raw_slots, a_bufs, d_bufs;
    unsigned idesc;
    Epilogue ep;
    const float* scales;           // 4-bit weights: [row block][stage][2][128]
    int* status;
    unsigned long long wait_limit_ns;
};

// D (CG x 128 rows x T columns) += A (rows x 16, tensor memory) x B (T x 16, shared memory of the CTAs)
template <int CG>
__device__ __forceinline__ void mma_from_tmem(unsigned d_tmem, unsigned a_tmem, unsigned long long bdesc, unsigned idesc, unsigned accumulate) {
    if constexpr (CG == 2) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
            ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
            : "memory");
    } else {
        tc_mma_ts(d_tmem, a_tmem, bdesc, idesc, accumulate);
    }
}
// nibbles n at bits [0,4) and [16,20) of w -> bf16x2 of (n - 8) * scale, each product rounded once from fp32
__device__ __forceinline__ unsigned nib2_to_bf16x2_scaled(unsigned w, f32x2 scale) {
    const unsigned a = nib2_to_bf16x2(w);
    float lo, hi;
    unpack2(mul2(pack2(__uint_as_float(a << 16), __uint_as_float(a & 0xffff0000u)), scale), lo, hi);
    return pack_bf16x2(lo, hi);
}
// Post-ops of 16 tokens of one output column n (the lane's weight row) and their stores.
struct RowVecs { float deq, bias, q; };
template <int KIND>
__device__ __forceinline__ void finish_chunk(float (&v)[CHUNK], int m, int n, const RowVecs& rv, const Epilogue& ep, int M, int n1) {
    char* dst = (char*)ep.C + (long long)m * ep.ldc;
    f32x2 w[CHUNK / 2];
#pragma unroll
    for (int j = 0; j < CHUNK / 2; j++) w[j] = mul2(pack2(v[2 * j], v[2 * j + 1]), pack2(rv.deq, rv.deq));
    if (ep.steps & B200FC_STEP_BIAS) {
#pragma unroll
        for (int j = 0; j < CHUNK / 2; j++) w[j] = add2(w[j], pack2(rv.bias, rv.bias));
    }
    if (ep.steps & B200FC_STEP_GELU) {
#pragma unroll
        for (int h = 0; h < CHUNK / 8; h++) {
            f32x2 t[4] = {w[4 * h], w[4 * h + 1], w[4 * h + 2], w[4 * h + 3]};
            gelu_erf_poly8(t);
#pragma unroll
            for (int j = 0; j < 4; j++) w[4 * h + j] = t[j];
        }
    }
    if (ep.steps & B200FC_STEP_QUANT) {
#pragma unroll
        for (int j = 0; j < CHUNK / 2; j++) w[j] = mul2(w[j], pack2(rv.q, rv.q));
    }
#pragma unroll
    for (int j = 0; j < CHUNK / 2; j++) unpack2(w[j], v[2 * j], v[2 * j + 1]);
    if (n >= n1) return;
#pragma unroll
    for (int t = 0; t < CHUNK; t++) {
        if (m + t >= M) break;
        if (ep.residual) v[t] += residual_at(ep, m + t, n);
        char* row = dst + t * ep.ldc;
        if constexpr (KIND == EPI_F32) ((float*)row)[n] = v[t];
        else if constexpr (KIND == EPI_BF16) ((unsigned short*)row)[n] = f32_to_bf16_bits(v[t]);
        else ((signed char*)row)[n] = (signed char)f32_to_s8(v[t]);
    }
}

template <int CG, int WB, int FOLD>
__global__ void __launch_bounds__(QT_THREADS, 1)
gemm_qt_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const QtParams p) {
    constexpr int PIECES = WB == 4 ? 2 : 1;           // pieces of 128 K per stored piece of 128 bytes
    constexpr int RAW_SLOT = RAW_BYTES + (WB == 4 ? 2 * QT_ROWS * 4 : 0);       // (with its 2 x 128 group scales)
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = smem_raw + (((smem_u32(smem_raw) + 1023u) & ~1023u) - smem_u32(smem_raw));
    const unsigned bars = smem_u32(smem + QT_RING);
    const unsigned bar_x_full = bars, bar_x_empty = bar_x_full + 8 * MAX_X;
    const unsigned bar_raw_full = bar_x_empty + 8 * MAX_X, bar_raw_empty = bar_raw_full + 8 * MAX_RAW;
    const unsigned bar_a_full = bar_raw_empty + 8 * MAX_RAW, bar_a_empty = bar_a_full + 8 * MAX_A;
    const unsigned bar_d_full = bar_a_empty + 8 * MAX_A, bar_d_empty = bar_d_full + 8 * MAX_D;
    unsigned* tmem_holder = (unsigned*)(smem + QT_RING + 16 * (MAX_X + MAX_RAW + MAX_A + MAX_D));
    volatile int* abort_flag = (volatile int*)(tmem_holder + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned crank = cluster_ctarank();
    const int rank = CG == 2 ? (int)(crank & 1) : 0;              // CTA of the pair
    const unsigned leader_rank = CG == 2 ? (crank & ~1u) : crank;
    const int split = CG == 2 ? (int)(crank >> 1) : (int)crank;
    const bool leader = rank == 0;
    const int unit = (int)(blockIdx.x / (unsigned)(CG * p.S)), units = (int)(gridDim.x / (unsigned)(CG * p.S));
    const int num_tiles = p.tiles_m * p.tiles_n;
    const int T = p.T, x_box = T / CG * SLAB_BYTES, x_slot = 2 * x_box;
    const int st0 = (int)((long long)p.stages * split / p.S), n_st = (int)((long long)p.stages * (split + 1) / p.S) - st0;
    const int n_pieces = n_st * PIECES;
    const int parts = FOLD ? min(p.parts, n_st) : 1;
    auto part_piece = [&](int q) { return FOLD ? n_st * q / parts * PIECES : q * n_pieces; };
    unsigned char* raw_ring = smem + p.x_slots * x_slot;
    const unsigned long long limit = p.wait_limit_ns;

    if (threadIdx.x == 0) {
        for (int i = 0; i < p.x_slots; i++) { mbar_init(bar_x_full + 8 * i, 1); mbar_init(bar_x_empty + 8 * i, 1); }
        for (int i = 0; i < p.raw_slots; i++) { mbar_init(bar_raw_full + 8 * i, 1); mbar_init(bar_raw_empty + 8 * i, 4 * PIECES); }
        for (int i = 0; i < p.a_bufs; i++) { mbar_init(bar_a_full + 8 * i, CG * 4); mbar_init(bar_a_empty + 8 * i, 1); }
        for (int i = 0; i < p.d_bufs; i++) { mbar_init(bar_d_full + 8 * i, 1); mbar_init(bar_d_empty + 8 * i, CG * QT_EPI_WARPS); }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        if constexpr (CG == 2) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_holder)), "r"(512u) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_holder)), "r"(512u) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();   // the pair's barriers exist before anyone signals them
    tc_fence_after();
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const unsigned tmem_base = *tmem_holder, tmem_d = tmem_base + p.a_bufs * A_COLS;

    if (warp == 0) {
        // ---------------- TMA: activations ----------------
        const unsigned leader_full = CG == 2 ? mapa_rank(bar_x_full, leader_rank) : bar_x_full;
        const unsigned tx = (unsigned)(CG * x_slot);
        asm volatile("griddepcontrol.wait;" ::: "memory");
        int slot = 0;
        unsigned phase = 0;
        bool alive = true;
        for (int tile = unit; tile < num_tiles && alive; tile += units) {
            const int row = tile % p.tiles_m * T + rank * (T / CG);
            for (int j = 0; j < n_pieces; j++) {
                alive = __all_sync(0xffffffffu, mbar_wait(bar_x_empty + 8 * slot, phase ^ 1, abort_flag, limit));
                if (!alive) break;
                if (elect_one()) {
                    const int k = (st0 * PIECES + j) * PIECE_K;
                    const unsigned dst = smem_u32(smem + slot * x_slot), full = leader_full + 8 * slot;
                    if (leader) mbar_expect_tx(bar_x_full + 8 * slot, tx);
                    if constexpr (CG == 2) {
                        tma_load_2d_pair(dst, &map_x, full, k, row);
                        tma_load_2d_pair(dst + x_box, &map_x, full, k + PIECE_K / 2, row);
                    } else {
                        tma_load_2d(dst, &map_x, full, k, row);
                        tma_load_2d(dst + x_box, &map_x, full, k + PIECE_K / 2, row);
                    }
                }
                if (++slot == p.x_slots) { slot = 0; phase ^= 1; }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ---------------- MMA issue ----------------
        if (leader) {
            int slot = 0, ab = 0, db = 0;
            unsigned phase = 0, a_phase = 0, d_phase = 0;
            bool alive = true;
            for (int tile = unit; tile < num_tiles && alive; tile += units) {
                for (int q = 0; q < parts && alive; q++) {
                    alive = __all_sync(0xffffffffu, mbar_wait<0, CG == 2>(bar_d_empty + 8 * db, d_phase ^ 1, abort_flag, limit));
                    if (!alive) break;
                    const int first = part_piece(q), end = part_piece(q + 1);
                    const unsigned d = tmem_d + (unsigned)(db * T);
                    for (int j = first; j < end; j++) {
                        alive = __all_sync(0xffffffffu, mbar_wait(bar_x_full + 8 * slot, phase, abort_flag, limit) &&
                                                            mbar_wait<0, CG == 2>(bar_a_full + 8 * ab, a_phase, abort_flag, limit));
                        if (!alive) break;
                        tc_fence_after();
                        const unsigned long long bdesc = make_smem_desc(smem_u32(smem + slot * x_slot));
                        const unsigned a = tmem_base + (unsigned)(ab * A_COLS);
                        if (elect_one()) {
#pragma unroll
                            for (int k = 0; k < 8; k++)
                                mma_from_tmem<CG>(d, a + k * 8, bdesc + (unsigned long long)((k >> 2) * (x_box >> 4) + (k & 3) * (MMA_K_BYTES >> 4)),
                                                  p.idesc, (unsigned)(j != first || k != 0));
                            if constexpr (CG == 2) {
                                const unsigned short mask = (unsigned short)(3u << leader_rank);
                                tc_commit_mask(bar_x_empty + 8 * slot, mask);
                                tc_commit_mask(bar_a_empty + 8 * ab, mask);
                                if (j == end - 1) tc_commit_mask(bar_d_full + 8 * db, mask);
                            } else {
                                tc_commit(bar_x_empty + 8 * slot);
                                tc_commit(bar_a_empty + 8 * ab);
                                if (j == end - 1) tc_commit(bar_d_full + 8 * db);
                            }
                        }
                        if (++slot == p.x_slots) { slot = 0; phase ^= 1; }
                        if (++ab == p.a_bufs) { ab = 0; a_phase ^= 1; }
                    }
                    if (++db == p.d_bufs) { db = 0; d_phase ^= 1; }
                }
            }
        }
        __syncwarp();
    } else if (warp == 2) {
        // ---------------- TMA: weights as stored; they do not depend on the previous kernel of the stream ----------------
        int slot = 0;
        unsigned phase = 0;
        bool alive = true;
        for (int tile = unit; tile < num_tiles && alive; tile += units) {
            const int row0 = p.n0 + (tile / p.tiles_m * CG + rank) * QT_ROWS;
            const int block = min(row0 / QT_ROWS, p.row_blocks - 1);       // (a pair's second block may lie past the matrix)
            for (int i = 0; i < n_st; i++) {
                alive = __all_sync(0xffffffffu, mbar_wait(bar_raw_empty + 8 * slot, phase ^ 1, abort_flag, limit));
                if (!alive) break;
                if (elect_one()) {
                    const unsigned dst = smem_u32(raw_ring + slot * RAW_SLOT), full = bar_raw_full + 8 * slot;
                    mbar_expect_tx(full, RAW_SLOT);
                    tma_load_2d(dst, &map_w, full, (st0 + i) * SLAB_BYTES, row0);
                    if constexpr (WB == 4)
                        bulk_load_1d(dst + RAW_BYTES, p.scales + ((size_t)block * p.stages + st0 + i) * (2 * QT_ROWS), RAW_SLOT - RAW_BYTES, full);
                }
                if (++slot == p.raw_slots) { slot = 0; phase ^= 1; }
            }
        }
        __syncwarp();
    } else if (warp >= FIRST_WIDENER) {
        // ---------------- widening ----------------
        const int set = (warp - FIRST_WIDENER) >> 2, quarter = warp & 3, row = quarter * 32 + lane, sw = row & 7;
        const unsigned a_base = tmem_base + ((unsigned)(quarter * 32) << 16);
        const unsigned leader_full = CG == 2 ? mapa_rank(bar_a_full, leader_rank) : bar_a_full;
        int half = 0, slot = 0, ab = 0;
        unsigned phase = 0, a_phase = 0;
        auto advance = [&]() {
            if (++half == PIECES) {
                half = 0;
                if (++slot == p.raw_slots) { slot = 0; phase ^= 1; }
            }
            if (++ab == p.a_bufs) { ab = 0; a_phase ^= 1; }
        };
        for (int i = 0; i < set; i++) advance();
        const int my_tiles = unit < num_tiles ? (num_tiles - unit + units - 1) / units : 0;
        const int total = my_tiles * n_pieces;
#pragma unroll 1
        for (int g = set; g < total; g += QT_SETS) {
            if (!__all_sync(0xffffffffu, mbar_wait(bar_raw_full + 8 * slot, phase, abort_flag, limit))) break;
            const unsigned char* src = raw_ring + slot * RAW_SLOT + row * SLAB_BYTES;
            bool alive = true;
#pragma unroll
            for (int h = 0; h < 2; h++) {              // 64 K each: 32 columns
                unsigned r[32];
                if constexpr (WB == 8) {
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        const uint4 v = *(const uint4*)(src + (((4 * h + u) ^ sw) << 4));
                        const unsigned w4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            r[8 * u + 2 * q] = u8x2_to_bf16x2_64th(w4[q], 0x4140);
                            r[8 * u + 2 * q + 1] = u8x2_to_bf16x2_64th(w4[q], 0x4342);
                        }
                    }
                } else {
                    const float sc1 = ((const float*)(raw_ring + slot * RAW_SLOT + RAW_BYTES))[half * QT_ROWS + row];
                    const f32x2 sc = pack2(sc1, sc1);
                    // K [32 j, +32) of group `half` lie in unit 2 j + half (see quant4_kernel in pack.cu)
#pragma unroll
                    for (int u = 0; u < 2; u++) {
                        const uint4 v = *(const uint4*)(src + (((2 * (2 * h + u) + half) ^ sw) << 4));
                        const unsigned w4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                        for (int q = 0; q < 4; q++)
#pragma unroll
                            for (int e = 0; e < 4; e++) r[16 * u + 4 * q + e] = nib2_to_bf16x2_scaled(w4[q] >> (4 * e), sc);
                    }
                }
                if (h == 0) {
                    alive = __all_sync(0xffffffffu, mbar_wait(bar_a_empty + 8 * ab, a_phase ^ 1, abort_flag, limit));
                    if (!alive) break;
                    tc_fence_after();
                }
                tc_st32(a_base + (unsigned)(ab * A_COLS + h * 32), r);
            }
            if (!alive) break;
            if (lane == 0) mbar_arrive(bar_raw_empty + 8 * slot);          // (every lane's bytes have gone through the stores above)
            tc_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                if (CG == 1 || leader) mbar_arrive(bar_a_full + 8 * ab);
                else mbar_arrive_leader(leader_full + 8 * ab);
            }
            for (int i = 0; i < QT_SETS; i++) advance();
        }
        __syncwarp();
    } else if (warp >= 4) {
        // ---------------- epilogue ----------------
        asm volatile("griddepcontrol.wait;" ::: "memory");
        const int quarter = warp & 3, half = (warp - 4) >> 2, row = quarter * 32 + lane, chunks = T / CHUNK;
        const unsigned lane_base = (unsigned)(quarter * 32) << 16;
        const unsigned leader_empty = CG == 2 ? mapa_rank(bar_d_empty, leader_rank) : bar_d_empty;
        const Epilogue& ep = p.ep;
        const int kind = ep.out_dtype == B200FC_F32 ? EPI_F32 : (ep.out_dtype == B200FC_BF16 ? EPI_BF16 : EPI_S8);
        int db = 0;
        unsigned d_phase = 0;
        bool ok = true;
        for (int tile = unit; tile < num_tiles && ok; tile += units) {
            const int n = p.n0 + (tile / p.tiles_m * CG + rank) * QT_ROWS + row, m0 = tile % p.tiles_m * T;
            RowVecs rv{1.0f, 0.0f, 1.0f};
            if (n < p.n1) {
                rv.deq = ep.deq_per_oc ? ep.deq_scale * __ldg(ep.deq_per_oc + n) : ep.deq_scale;
                if (ep.steps & B200FC_STEP_BIAS) rv.bias = __ldg(ep.bias + n);
                if (ep.steps & B200FC_STEP_QUANT) rv.q = ep.q_per_oc ? __ldg(ep.q_per_oc + n) : ep.q_scale;
            }
            float sum[FOLD ? FOLD / CHUNK / QT_EPI_SETS : 1][CHUNK];
            auto load_acc = [&](int c, float (&v)[CHUNK]) {
                unsigned r[CHUNK];
                __syncwarp();
                tc_ld16(tmem_d + lane_base + (unsigned)(db * T + c * CHUNK), r);
                tc_wait_ld();
#pragma unroll
                for (int t = 0; t < CHUNK; t++) v[t] = __uint_as_float(r[t]) * (WB == 8 ? 64.0f : 1.0f);       // (int8: the weights are in 64ths)
            };
            auto release = [&]() {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    if (CG == 1 || leader) mbar_arrive(bar_d_empty + 8 * db);
                    else mbar_arrive_remote(leader_empty + 8 * db);
                }
                if (++db == p.d_bufs) { db = 0; d_phase ^= 1; }
            };
            auto wait_acc = [&]() {
                ok = __all_sync(0xffffffffu, mbar_wait<32>(bar_d_full + 8 * db, d_phase, abort_flag, limit));
                tc_fence_after();
            };
            if constexpr (FOLD > 0) {
                // all parts into registers, in order
#pragma unroll
                for (int i = 0; i < FOLD / CHUNK / QT_EPI_SETS; i++)
#pragma unroll
                    for (int t = 0; t < CHUNK; t++) sum[i][t] = 0.0f;
                for (int q = 0; q < parts; q++) {
                    wait_acc();
                    if (!ok) break;
#pragma unroll
                    for (int i = 0; i < FOLD / CHUNK / QT_EPI_SETS; i++) {
                        if (QT_EPI_SETS * i + half < chunks) {
                            float v[CHUNK];
                            load_acc(QT_EPI_SETS * i + half, v);
#pragma unroll
                            for (int t = 0; t < CHUNK; t++) sum[i][t] += v[t];
                        }
                    }
                    release();
                }
            } else {
                wait_acc();
            }
            // body(chunk, its sums) over this warp's chunks of the tile
            auto each_chunk = [&](auto&& body) {
                if constexpr (FOLD > 0) {
#pragma unroll
                    for (int i = 0; i < FOLD / CHUNK / QT_EPI_SETS; i++)
                        if (QT_EPI_SETS * i + half < chunks) body(QT_EPI_SETS * i + half, sum[i]);
                } else {
#pragma unroll 1
                    for (int c = half; c < chunks; c += QT_EPI_SETS) {
                        float v[CHUNK];
                        load_acc(c, v);
                        body(c, v);
                    }
                }
            };
            auto finish = [&](int c, float (&v)[CHUNK]) {
                const int m = m0 + c * CHUNK;
                if (m >= p.M) return;
                switch (kind) {
                    case EPI_F32: finish_chunk<EPI_F32>(v, m, n, rv, ep, p.M, p.n1); break;
                    case EPI_BF16: finish_chunk<EPI_BF16>(v, m, n, rv, ep, p.M, p.n1); break;
                    default: finish_chunk<EPI_S8>(v, m, n, rv, ep, p.M, p.n1); break;
                }
            };
            if (p.S == 1) {
                if (ok) each_chunk(finish);
            } else {
                // (one tile) Part `split` of K hands chunk c of its sums to part (c mod S) of the cluster: posted stores into its ring,
                // which every MMA of the cluster has left
                const unsigned mine = smem_u32(smem) + (unsigned)(row * 16);
                __syncwarp();
                cluster_sync_all();
                if (ok)
                    each_chunk([&](int c, float (&v)[CHUNK]) {
                        const unsigned dst = mapa_rank(mine + (unsigned)((c / p.S * p.S + split) * CHUNK_BYTES), (unsigned)(c % p.S * CG + rank));
#pragma unroll
                        for (int j = 0; j < CHUNK / 4; j++)
                            st_cluster_v4(dst + (unsigned)(j * QT_ROWS * 16), __float_as_uint(v[4 * j]), __float_as_uint(v[4 * j + 1]),
                                          __float_as_uint(v[4 * j + 2]), __float_as_uint(v[4 * j + 3]));
                    });
                __syncwarp();
                cluster_sync_all();
#pragma unroll 1
                for (int t = half, c = split + half * p.S; ok && c < chunks; t += QT_EPI_SETS, c += QT_EPI_SETS * p.S) {
                    const float4* src = (const float4*)(smem + t * p.S * CHUNK_BYTES) + row;
                    float v[CHUNK];
#pragma unroll
                    for (int j = 0; j < CHUNK; j++) v[j] = 0.0f;
#pragma unroll 2
                    for (int q = 0; q < p.S; q++)
#pragma unroll
                        for (int j = 0; j < CHUNK / 4; j++) {
                            const float4 x = src[q * (CHUNK_BYTES / 16) + j * QT_ROWS];
                            v[4 * j] += x.x; v[4 * j + 1] += x.y; v[4 * j + 2] += x.z; v[4 * j + 3] += x.w;
                        }
                    finish(c, v);
                }
            }
            if (!FOLD && ok) release();
        }
        __syncwarp();
    }
    if ((warp < 4 || warp >= FIRST_WIDENER) && p.S > 1) {
        __syncwarp();
        cluster_sync_all();   // (the epilogue's barriers around the exchange of partial sums)
        cluster_sync_all();
    }

    // ---------------- common exit ----------------
    tc_fence_before();
    __syncthreads();
    if (*abort_flag) {
        if (threadIdx.x == 0) {
            atomicExch(p.status, 2);
            const unsigned long long t0 = globaltimer();
            while (globaltimer() - t0 < 200000ull) { }   // copies still in flight land before shared memory is released
        }
        __syncthreads();
    }
    cluster_sync_all();   // a peer may still signal this CTA's barriers or read its partial sums until here
    if (warp == 1) {
        tc_fence_after();
        if constexpr (CG == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    }
}

// ---- host side ----------------------------------------------------------------------------------------------------------
struct QtShape { int cg, T, S, units, parts; };

template <int CG>
int max_units(int S, int* out) {
    static ClusterCounts counts;
    int n = 0;
    const int rc = resident_clusters(counts, CG * S, QT_THREADS, QT_SMEM, &n);
    if (rc) return rc;
    const int by_sms = num_sms() / (CG * S);
    *out = n < by_sms ? n : by_sms;
    return B200FC_OK;
}

int d_bufs(int T) { return 2 * T <= 512 - QT_SETS * A_COLS ? 2 : 1; }       // accumulators beside the A buffers in tensor memory

// Picks pairs or single CTAs, the tokens of a tile and the split of K by a model of SM clocks, fitted to 1000 timed shapes of 74 calls
// (8 % rms; the calls lose 2 % on average against their best shape).  A piece costs the loads (38 bytes per clock and SM come from L2 in
// pairs, 49 in single CTAs), or the MMAs (4 clocks per token) and the widening (690 clocks int8, 930 4 bits), which get in each
// other's way: the root of the sum of their squares.  Then HBM, the epilogue (of every tile where tensor memory holds one accumulator
// only, or where it is longer than a tile's pieces) and the exchange of the parts of K.
template <int CG, int WB>
int consider(int M, int nspan, int stages, int chains, bool even, bool one_chain, QtShape* best, double* best_cost) {
    constexpr int PIECES = WB == 4 ? 2 : 1;
    const int tiles_n = (nspan + CG * QT_ROWS - 1) / (CG * QT_ROWS), max_S = one_chain ? 1 : 8 / CG;
    for (int S = 1; S <= max_S && S <= stages; S++) {
        int units = 0;
        const int rc = max_units<CG>(S, &units);
        if (rc) return rc;
        const int parts = parts_of_share(stages, S, chains, even);
        for (int T = 16 * CG; T <= 256; T += 16 * CG) {
            if (T / CG > 128 || (parts > 1 && T > 192)) continue;
            const int tiles_m = (M + T - 1) / T;
            if (T > 16 * CG && (M + T - 16 * CG - 1) / (T - 16 * CG) == tiles_m) continue;       // a smaller tile does as well
            const long long tiles = (long long)tiles_m * tiles_n;
            if (S > 1 && tiles > units) continue;
            const int rounds = (int)((tiles + units - 1) / units);
            const double load = (T / CG * 256.0 + RAW_BYTES / PIECES) / (CG == 2 ? 38.0 : 49.0), mma = 4.0 * T, cvt = WB == 4 ? 930.0 : 690.0;
            const double product = sqrt(mma * mma + cvt * cvt), piece = load > product ? load : product;
            const double tile = piece * ((stages + S - 1) / S * PIECES);
            const double epi = 6490.0 + 41.0 * T + (parts > 1 && T > 128 ? 30.0 * T : 0.0);
            double loop = tile * rounds;
            if (d_bufs(T) == 1) loop += epi * (rounds - 1);
            else if (epi > tile) loop += (epi - tile) * (rounds - 1);
            const double hbm = (double)nspan * stages * SLAB_BYTES / 2230.0;
            if (loop < hbm) loop = hbm;
            const double cost = 2170.0 + loop + epi + (S > 1 ? 2910.0 + 2.2 * T : 0.0);
            if (*best_cost < 0 || cost < *best_cost) {
                *best_cost = cost;
                *best = QtShape{CG, T, S, (int)(tiles < units ? tiles : units), parts};
            }
        }
    }
    return B200FC_OK;
}

struct QtCall {
    const Weight& w;
    const void* A;
    int M, K;
    int64_t lda;
    int n0, n1;
    const Epilogue& ep;
    cudaStream_t s;
};

template <int CG, int WB, int FOLD>
int run_qt(const QtCall& call, const QtShape& sh) {
    constexpr int RAW_SLOT = RAW_BYTES + (WB == 4 ? 2 * QT_ROWS * 4 : 0);
    static std::atomic<unsigned long long> attr_devices{0};
    int rc = once_per_device(attr_devices, [] {
        B200FC_CUDA(cudaFuncSetAttribute(gemm_qt_kernel<CG, WB, FOLD>, cudaFuncAttributeMaxDynamicSharedMemorySize, QT_SMEM));
        return (int)B200FC_OK;
    });
    if (rc) return rc;
    QtParams p = {};
    p.M = call.M; p.n0 = call.n0; p.n1 = call.n1; p.row_blocks = call.w.N_pad / QT_ROWS;
    p.T = sh.T; p.S = sh.S; p.parts = sh.parts;
    p.tiles_m = (call.M + sh.T - 1) / sh.T;
    p.tiles_n = (call.n1 - call.n0 + CG * QT_ROWS - 1) / (CG * QT_ROWS);
    p.stages = (int)(call.w.ld_bytes() / SLAB_BYTES);
    const int x_slot = sh.T / CG * 2 * SLAB_BYTES;
    // A set of widening warps does not see every phase of a barrier, and the parity of a wait is only right while the barrier is at most one
    // phase behind: a_bufs >= sets (the set's previous piece waited for the MMAs of a piece at least that recent), and raw_slots a
    // multiple of the sets (int8: a set always comes back to the same slots; 4 bits: two sets see every slot).
    p.raw_slots = 4;
    p.x_slots = (QT_RING - p.raw_slots * RAW_SLOT) / x_slot;
    if (p.x_slots > MAX_X) p.x_slots = MAX_X;
    p.d_bufs = d_bufs(sh.T);
    p.a_bufs = (512 - p.d_bufs * sh.T) / A_COLS;
    if (p.a_bufs > MAX_A) p.a_bufs = MAX_A;
    p.idesc = make_idesc(false, false, false, sh.T, CG * BM);
    p.ep = call.ep;
    if (!(p.ep.steps & B200FC_STEP_DEQUANT)) { p.ep.deq_scale = 1.0f; p.ep.deq_per_oc = nullptr; }
    p.scales = call.w.scale_grp;
    p.status = kernel_status_word();
    if (!p.status) { set_error("gemm: no kernel status word on this device"); return B200FC_ERR_CUDA; }
    p.wait_limit_ns = wait_limit_ns();
    CUtensorMap mx, mw;
    rc = make_map(&mx, call.A, false, (uint64_t)call.K, (uint64_t)call.M, (uint64_t)call.lda, (uint32_t)(sh.T / CG));
    if (rc) return rc;
    rc = make_map(&mw, call.w.data, true, (uint64_t)call.w.ld_bytes(), (uint64_t)call.w.N_pad, (uint64_t)call.w.ld_bytes(), QT_ROWS);
    if (rc) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(CG * sh.S * sh.units), 1, 1);
    cfg.blockDim = dim3(QT_THREADS, 1, 1);
    cfg.dynamicSmemBytes = QT_SMEM;
    cfg.stream = call.s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)(CG * sh.S);
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    B200FC_CUDA(cudaLaunchKernelEx(&cfg, gemm_qt_kernel<CG, WB, FOLD>, mx, mw, p));
    count_launch();
    return B200FC_OK;
}

template <int WB>
int run_qt(const QtCall& c, int chains, bool even) {
    const int stages = (int)(c.w.ld_bytes() / SLAB_BYTES);
    QtShape sh = {};
    double cost = -1.0;
    const bool one_chain = WB == 8 && sums_pinned(c.ep);      // (the caller sends such calls only with chains = 1)
    int rc = consider<1, WB>(c.M, c.n1 - c.n0, stages, chains, even, one_chain, &sh, &cost);
    if (rc) return rc;
    rc = consider<2, WB>(c.M, c.n1 - c.n0, stages, chains, even, one_chain, &sh, &cost);
    if (rc) return rc;
    // (FOLD: the most tokens whose sums a call keeps.  Those of 192 spill, which costs small tiles: 4 bits 100 x 4096 x 11008 34 us instead of 27;
    // but wider tiles are worth it: 493 x 7680 x 14848 116 us, 132 with 128.)
    if (sh.parts > 1) return sh.cg == 1 ? run_qt<1, WB, 128>(c, sh) : sh.T <= 128 ? run_qt<2, WB, 128>(c, sh) : run_qt<2, WB, 192>(c, sh);
    return sh.cg == 1 ? run_qt<1, WB, 0>(c, sh) : run_qt<2, WB, 0>(c, sh);
}

}  // namespace

int launch_gemm_qt(const Weight& w, const void* A, int M, int K, int64_t lda, int n0, int n1, const Epilogue& ep, int chains, bool even, cudaStream_t s) {
    if (M <= 0 || n1 <= n0) return B200FC_OK;
    const QtCall c{w, A, M, K, lda, n0, n1, ep, s};
    return w.dtype == B200FC_S4 ? run_qt<4>(c, chains, even) : run_qt<8>(c, chains, even);
}

}  // namespace b200fc
