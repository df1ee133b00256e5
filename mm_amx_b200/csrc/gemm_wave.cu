// Fully-connected layer whose output fits the GPU as ONE wave of tiles: small and medium prefill calls (17 rows and more).
//
// Replaces the same M > 16 branches as gemm_tc.cu (include/kernels_amx.hpp:1255-1313), and those of the compressed-weight
// specialisation (kernels_amx.hpp:1443-1514).  gemm_tc.cu's kernel is persistent over tiles of a fixed width, which pays
// for its double-buffered accumulators once every SM has several tiles; a call with about as many tiles as SMs loses most of
// its time to a ragged second round, to a split of K that goes through global memory, and (quantised weights) to a pass
// that widens the weights to bf16 before anything is multiplied.  Here:
//   - every CTA, or pair of CTAs (more than 128 rows), gets exactly one tile of 128 / 256 rows x W columns, W any multiple
//     of 32 / 64 up to 256 / 512 (all of TMEM): the launcher picks W and the split of K so that one wave fills the SMs;
//   - the S parts of a split K form one cluster and add their accumulators in rank order through distributed shared memory;
//   - int8-compressed and 4-bit weights cross HBM and L2 as they are stored: twelve warps widen each slab to bf16 in shared
//     memory between the TMA load and the MMA.  (Most calls with such weights go to gemm_qt.cu, see run_wave.)
// int8 values are exact in bf16; a 4-bit value is multiplied by its group scale in fp32 and rounded to bf16.
//
// Warps: 0 = TMA loads of activations (and of plain weights), 1 = MMA issue (one lane) and TMEM owner, 2 = TMA loads of
// quantised weights, 3 idle, 4-15 = widening, then epilogue (three warps per TMEM quarter).
// Rings: slots of activations and plain weights (full[s] in the pair's leader: one arrive.expect_tx for the bytes of both CTAs;
// empty[s] in each CTA, released by the leader's tcgen05.commit); quantised weights have a ring of their own for the widened
// slabs (wide_full: the arrivals of the widening warps of both CTAs that take the slab), so that the activations' ring can
// be deep enough for their latency, and a third one for the pieces as stored (raw).  Every wait is bounded as in gemm_tc.cu.
#include <cstdlib>
#include "tc_common.cuh"

namespace b200fc {

namespace {

// weights: bf16, 8-bit (8-bit MMA), int8 compressed, 4-bit; W_I8_HALF: 8-bit whose int8 output rows are 8-byte aligned only (inside the
// 8-bit kernel its epilogue costs the others registers: 2048 x 4096 x 4096 33.44 us instead of 33.26)
enum WaveMode { W_BF16 = 0, W_I8 = 1, W_U8C = 2, W_U4C = 3, W_I8_HALF = 4 };

constexpr int SETS = 3;                               // sets of four worker warps, one warp of a set per TMEM quarter
constexpr int WORKERS = 4 * SETS;
constexpr int WAVE_THREADS = 128 + 32 * WORKERS;
constexpr int MAX_SLOTS = 12, MAX_RAW = 8, MAX_WIDE = 4, MAX_W = 512;
constexpr int WAVE_BAR_BYTES = 512;
constexpr int COLVEC_FLOATS = 3 * MAX_W;
constexpr int WAVE_SMEM = 232448;                                                  // all an SM gives to one CTA
constexpr int RING_BYTES = (WAVE_SMEM - 1024 - WAVE_BAR_BYTES - COLVEC_FLOATS * 4) / 1024 * 1024;
constexpr int CHUNK_BYTES = 32 * BM * 4;                                           // 32 columns of fp32 / int32 partial sums
constexpr int WARP_TILE_BYTES = 4096;                                              // staging tile of an epilogue warp

struct WaveParams {
    int M, n0, n1, n_pad;
    int R, R0;              // weight rows (= output columns) per CTA; of the first MMA of a K step
    int tiles_m, S;
    int parts, sets;        // parts of a CTA's K, and accumulators that the slabs of a part take in turn (W columns of tensor memory each)
    char* sums;             // what the parts but the last add up to: a tile of 128 rows x W columns per CTA, or null (one part)
    int slabs, units;       // K in 128-byte slabs of the MMA operands / in 128-byte pieces of the stored weight rows
    int slots, raw_slots, wide_slots;
    unsigned idesc0, idesc1;
    int vec_ok;
    Epilogue ep;
    const float* scale_grp;
    int* status;
    unsigned long long wait_limit_ns;
};

// nibbles n at bits [0,4) and [16,20) of w -> bf16x2 of (n - 8) * scale, each product rounded once from fp32
__device__ __forceinline__ unsigned nib2_to_bf16x2_scaled(unsigned w, float scale) {
    const unsigned a = nib2_to_bf16x2(w);
    const __nv_bfloat162 r = __floats2bfloat162_rn(__uint_as_float(a << 16) * scale, __uint_as_float(a & 0xffff0000u) * scale);
    return *(const unsigned*)&r;
}

// FOLD: K in several parts, see below (quantised weights).  A kernel of its own, because the folding code costs the widening loop
// registers and instruction cache also where it does not run (int8 705 x 2560 x 10240: 44.8 us with it, 42.3 without).  Calls whose
// chains do not fit pay for both (us, one chain / as many as asked for / through widened blocks and a split of K): 4 bits
// 512 x 4096 x 11008 42 / 62 / 127 (two folds), int8 705 x 4096 x 10240 45 / 59 / 126 (one fold, 6.5 of it, of which the workers read
// tensor memory at 500 clocks per 32 columns), int8 300 x 11008 x 8192 74 / 99 / 249.  Parts that end anywhere, with the check for a
// fold inside the loop over a piece's slabs: 66 / 59 / 102.  No gain: folding each chain by itself under the next one, adding with
// red instead of load and store, the fold as a function that is called.
template <int CG, int MODE, bool FOLD>
__global__ void __launch_bounds__(WAVE_THREADS, 1)
gemm_wave_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, const WaveParams p) {
    constexpr bool I8 = MODE == W_I8 || MODE == W_I8_HALF, WQ = MODE == W_U8C || MODE == W_U4C;
    constexpr int SPU = MODE == W_U8C ? 2 : (MODE == W_U4C ? 4 : 1);   // slabs per stored 128-byte piece
    constexpr int A_BYTES = BM * SLAB_BYTES;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = smem_raw + (((smem_u32(smem_raw) + 1023u) & ~1023u) - smem_u32(smem_raw));
    const unsigned bars = smem_u32(smem + RING_BYTES);
    const unsigned bar_full = bars, bar_empty = bars + 8 * MAX_SLOTS;
    const unsigned bar_raw_full = bars + 16 * MAX_SLOTS, bar_raw_empty = bar_raw_full + 8 * MAX_RAW;
    const unsigned bar_wide_full = bar_raw_empty + 8 * MAX_RAW, bar_wide_empty = bar_wide_full + 8 * MAX_WIDE;
    const unsigned bar_acc = bar_wide_empty + 8 * MAX_WIDE, bar_part = bar_acc + 8, bar_folded = bar_part + 8;
    unsigned* tmem_holder = (unsigned*)(smem + RING_BYTES + 16 * (MAX_SLOTS + MAX_RAW + MAX_WIDE) + 24);
    volatile int* abort_flag = (volatile int*)(tmem_holder + 1);
    float* colvec = (float*)(smem + RING_BYTES + WAVE_BAR_BYTES);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned crank = cluster_ctarank();
    const int rank = CG == 2 ? (int)(crank & 1) : 0;        // CTA of the pair
    const unsigned leader_rank = CG == 2 ? (crank & ~1u) : crank;
    const int split = CG == 2 ? (int)(crank >> 1) : (int)crank;
    const bool leader = rank == 0;
    const int tile = (int)(blockIdx.x / (unsigned)(CG * p.S));
    const int tm = tile % p.tiles_m, tn = tile / p.tiles_m;
    const int W = CG * p.R, nb = p.n0 + tn * W;
    const int w_bytes = p.R * SLAB_BYTES;                          // a slab of weights as MMA operand; a stored piece of as many rows
    const int stage_bytes = A_BYTES + (WQ ? 0 : w_bytes);
    unsigned char* wide_ring = smem + p.slots * stage_bytes;
    unsigned char* raw_ring = wide_ring + p.wide_slots * w_bytes;
    const int u0 = (int)((long long)p.units * split / p.S), u1 = (int)((long long)p.units * (split + 1) / p.S);
    const int n_units = u1 - u0, n_slabs = min(u1 * SPU, p.slabs) - u0 * SPU;
    // K in chains of fp32 sums: the slabs take the accumulators in turn.  Where tensor memory holds too few of them K is cut into parts
    // as well, after each of which (but the last) the workers add the accumulators to a sum in global memory (L2).
    // Parts end with stored pieces, so that the folding stays out of the loop over a piece's slabs.
    const int parts = FOLD ? min(p.parts, n_units) : 1, cols = p.sets * W;
    auto part_unit = [&](int q) { return n_units * q / parts; };
    auto part_slab = [&](int q) { return FOLD ? min(part_unit(q) * SPU, n_slabs) : q * n_slabs; };
    const unsigned tmem_cols = cols <= 32 ? 32 : (cols <= 64 ? 64 : (cols <= 128 ? 128 : (cols <= 256 ? 256 : 512)));

    if (threadIdx.x == 0) {
        for (int i = 0; i < p.slots; i++) {
            mbar_init(bar_full + 8 * i, 1);
            mbar_init(bar_empty + 8 * i, 1);
        }
        for (int i = 0; i < p.raw_slots; i++) {
            mbar_init(bar_raw_full + 8 * i, 1);
            mbar_init(bar_raw_empty + 8 * i, WORKERS);
        }
        for (int i = 0; i < p.wide_slots; i++) {
            mbar_init(bar_wide_full + 8 * i, CG * 4);
            mbar_init(bar_wide_empty + 8 * i, 1);
        }
        mbar_init(bar_acc, 1);
        mbar_init(bar_part, 1);
        mbar_init(bar_folded, CG * WORKERS);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        if constexpr (CG == 2) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_holder)), "r"(tmem_cols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_holder)), "r"(tmem_cols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();   // the pair's barriers exist before anyone signals them
    tc_fence_after();
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const unsigned tmem_base = *tmem_holder;

    if (warp == 0) {
        // ---------------- TMA: activations, and weights that need no widening ----------------
        const unsigned leader_full = CG == 2 ? mapa_rank(bar_full, leader_rank) : bar_full;
        const int row_a = (tm * CG + rank) * BM, row_w = nb + rank * p.R;
        const unsigned tx = (unsigned)(CG * stage_bytes);
        const unsigned ring = smem_u32(smem);
        auto load_a = [&](int ks, int slot) {
            const int kx = ks * (I8 ? SLAB_BYTES : SLAB_BYTES / 2);
            const unsigned dst = ring + (unsigned)(slot * stage_bytes);
            if constexpr (CG == 2) tma_load_2d_pair(dst, &map_a, leader_full + 8 * slot, kx, row_a);
            else tma_load_2d(dst, &map_a, leader_full + 8 * slot, kx, row_a);
        };
        auto load_w = [&](int ks, int slot) {
            const int kx = ks * (I8 ? SLAB_BYTES : SLAB_BYTES / 2);
            const unsigned dst = ring + (unsigned)(slot * stage_bytes) + A_BYTES;
            if constexpr (CG == 2) tma_load_2d_pair(dst, &map_w, leader_full + 8 * slot, kx, row_w);
            else tma_load_2d(dst, &map_w, leader_full + 8 * slot, kx, row_w);
        };
        // plain weights do not depend on the previous kernel of the stream: the first ring of them travels while it ends
        const int pre = WQ ? 0 : min(p.slots, n_units);
        for (int j = 0; j < pre; j++)
            if (elect_one()) {
                if (leader) mbar_expect_tx(bar_full + 8 * j, tx);
                load_w(u0 + j, j);
            }
        asm volatile("griddepcontrol.wait;" ::: "memory");
        int slot = 0;
        unsigned phase = 0;
        bool alive = true;
        for (int j = 0; j < n_units && alive; j++) {
            const int ks_first = (u0 + j) * SPU;
            for (int ks = ks_first; ks < min(ks_first + SPU, p.slabs); ks++) {
                if (j >= pre) {
                    alive = __all_sync(0xffffffffu, mbar_wait(bar_empty + 8 * slot, phase ^ 1, abort_flag, p.wait_limit_ns));
                    if (!alive) break;
                }
                if (elect_one()) {
                    if (j >= pre) {
                        if (leader) mbar_expect_tx(bar_full + 8 * slot, tx);
                        if (!WQ) load_w(ks, slot);
                    }
                    load_a(ks, slot);
                }
                if (++slot == p.slots) { slot = 0; phase ^= 1; }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ---------------- MMA issue ----------------
        if (leader) {
            int slot = 0, wslot = 0, set = 0, part = 0, start = 0, end = part_slab(1);      // slabs of the part
            unsigned phase = 0, wphase = 0;
            const unsigned ring = smem_u32(smem), wring = smem_u32(wide_ring);
            for (int i = 0; i < n_slabs; i++) {
                if (FOLD && i == end) {
                    if (!__all_sync(0xffffffffu, mbar_wait<0, CG == 2>(bar_folded, (unsigned)part & 1, abort_flag, p.wait_limit_ns))) break;
                    part++;
                    start = end;
                    end = part_slab(part + 1);
                    set = 0;
                }
                if (!__all_sync(0xffffffffu, mbar_wait(bar_full + 8 * slot, phase, abort_flag, p.wait_limit_ns))) break;
                if (WQ && !__all_sync(0xffffffffu, mbar_wait<0, CG == 2>(bar_wide_full + 8 * wslot, wphase, abort_flag, p.wait_limit_ns))) break;
                tc_fence_after();
                const unsigned sa = ring + (unsigned)(slot * stage_bytes);
                const unsigned sb = WQ ? wring + (unsigned)(wslot * w_bytes) : sa + A_BYTES;
                const unsigned long long adesc = make_smem_desc(sa);
                const unsigned long long bdesc = make_smem_desc(sb);
                const unsigned long long bdesc1 = make_smem_desc(sb + p.R0 * SLAB_BYTES);
                if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < SLAB_BYTES / MMA_K_BYTES; k++) {
                        const unsigned long long adv = (unsigned long long)(k * (MMA_K_BYTES >> 4));
                        const unsigned acc = (unsigned)(i - start >= p.sets || k != 0);
                        if constexpr (CG == 2) tc_mma_pair<I8>(tmem_base + set * W, adesc + adv, bdesc + adv, p.idesc0, acc);
                        else tc_mma<I8>(tmem_base + set * W, adesc + adv, bdesc + adv, p.idesc0, acc);
                        if (CG == 2 && p.R0 < p.R) tc_mma_pair<I8>(tmem_base + set * W + 2 * p.R0, adesc + adv, bdesc1 + adv, p.idesc1, acc);
                    }
                    if constexpr (CG == 2) {
                        const unsigned short mask = (unsigned short)(3u << leader_rank);
                        tc_commit_mask(bar_empty + 8 * slot, mask);
                        if (WQ) tc_commit_mask(bar_wide_empty + 8 * wslot, mask);
                        if (FOLD && i == end - 1 && i != n_slabs - 1) tc_commit_mask(bar_part, mask);
                        if (i == n_slabs - 1) tc_commit_mask(bar_acc, mask);
                    } else {
                        tc_commit(bar_empty + 8 * slot);
                        if (WQ) tc_commit(bar_wide_empty + 8 * wslot);
                        if (FOLD && i == end - 1 && i != n_slabs - 1) tc_commit(bar_part);
                        if (i == n_slabs - 1) tc_commit(bar_acc);
                    }
                }
                if (++set == p.sets) set = 0;
                if (++slot == p.slots) { slot = 0; phase ^= 1; }
                if (WQ && ++wslot == p.wide_slots) { wslot = 0; wphase ^= 1; }
            }
        }
        __syncwarp();
    } else if (warp == 2) {
        // ---------------- TMA: quantised weights as stored ----------------
        if (WQ) {
            int slot = 0;
            unsigned phase = 0;
            for (int j = 0; j < n_units; j++) {
                const int u = u0 + j;
                if (!__all_sync(0xffffffffu, mbar_wait(bar_raw_empty + 8 * slot, phase ^ 1, abort_flag, p.wait_limit_ns))) break;
                if (elect_one()) {
                    mbar_expect_tx(bar_raw_full + 8 * slot, (unsigned)w_bytes);
                    tma_load_2d(smem_u32(raw_ring + slot * w_bytes), &map_w, bar_raw_full + 8 * slot, u * SLAB_BYTES, nb + rank * p.R);
                }
                if (++slot == p.raw_slots) { slot = 0; phase ^= 1; }
            }
        }
        __syncwarp();
    } else if (warp >= 4) {
        const int wi = warp - 4;
        bool ok = true;
        // per-column vectors of the tile (they may come from the previous kernel of the stream)
        asm volatile("griddepcontrol.wait;" ::: "memory");
        const bool plain_ep = !(p.ep.steps & B200FC_STEP_SILU_MUL) && p.ep.out_dtype != B200FC_S32;
        const bool use_deq = plain_ep && (p.ep.steps & B200FC_STEP_DEQUANT) && p.ep.deq_per_oc;
        const bool use_bias = plain_ep && (p.ep.steps & B200FC_STEP_BIAS) && p.ep.bias;
        const bool use_q = plain_ep && (p.ep.steps & B200FC_STEP_QUANT) && p.ep.q_per_oc;
        if (use_deq || use_bias || use_q)
            for (int i = wi * 32 + lane; i < W; i += WORKERS * 32) {
                const int col = min(nb + i, p.n1 - 1);
                if (use_deq) colvec[i] = __ldg(p.ep.deq_per_oc + col);
                if (use_bias) colvec[MAX_W + i] = __ldg(p.ep.bias + col);
                if (use_q) colvec[2 * MAX_W + i] = __ldg(p.ep.q_per_oc + col);
            }
        const int quarter = warp & 3, third = wi >> 2;
        const int chunks = W / 32;
        const unsigned taddr = tmem_base + ((unsigned)(quarter * 32) << 16);
        // this thread's row of a chunk's sums: eight 16-byte units, one per four columns; only this thread reads and writes them
        auto sums_of = [&](int c) {
            return (uint4*)(p.sums + ((size_t)blockIdx.x * chunks + c) * CHUNK_BYTES) + quarter * 32 + lane;
        };
        auto load_sums = [&](int c, unsigned (&r)[32]) {
            const uint4* src = sums_of(c);
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const uint4 v = __ldcg(src + j * BM);
                r[4 * j] = v.x; r[4 * j + 1] = v.y; r[4 * j + 2] = v.z; r[4 * j + 3] = v.w;
            }
        };
        // the accumulators of a part, once its MMAs are done, into the sums: fp32 adds in order, the columns shared out as in the epilogue
        const unsigned folded_leader = CG == 2 ? mapa_rank(bar_folded, leader_rank) : bar_folded;
        int folds = 0;
        auto fold_part = [&]() {
            ok = __all_sync(0xffffffffu, mbar_wait(bar_part, (unsigned)folds & 1, abort_flag, p.wait_limit_ns));
            if (!ok) return;
            tc_fence_after();
            const int filled = min(p.sets, part_slab(folds + 1) - part_slab(folds));
#pragma unroll 1
            for (int c = third; c < chunks; c += SETS) {
                unsigned sum[32], x[32];
                if (folds) {
                    load_sums(c, sum);
                } else {
                    tc_ld32(taddr + (unsigned)(c * 32), sum);
                    tc_wait_ld();
                }
#pragma unroll 1
                for (int t = folds ? 0 : 1; t < filled; t++) {
                    tc_ld32(taddr + (unsigned)(t * W + c * 32), x);
                    tc_wait_ld();
#pragma unroll
                    for (int j = 0; j < 32; j++) sum[j] = __float_as_uint(__uint_as_float(sum[j]) + __uint_as_float(x[j]));
                }
                uint4* dst = sums_of(c);
#pragma unroll
                for (int j = 0; j < 8; j++) __stcg(dst + j * BM, make_uint4(sum[4 * j], sum[4 * j + 1], sum[4 * j + 2], sum[4 * j + 3]));
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                if (CG == 1 || leader) mbar_arrive(bar_folded);
                else mbar_arrive_remote(folded_leader);
            }
            folds++;
        };
        if constexpr (WQ) {
            // ---------------- widening ----------------
            // The sets of four warps take the slabs in turn, so that a warp's waits, its proxy fence and its arrival (about
            // a thousand clocks, mostly latency) come once per SETS slabs.  Inside a slab a warp takes every fourth item; an
            // item is 32 rows (one per lane) x 32 K, read before the slot is waited for.
            const int set = wi >> 2, w_in_set = wi & 3, n_items = p.R / 16;
            const unsigned leader_full = CG == 2 ? mapa_rank(bar_wide_full, leader_rank) : bar_wide_full;
            // 4-bit weights: the scales of this thread's rows for the two groups of 128 K of a piece, one piece ahead
            float sc[4][2] = {}, sc_next[4][2] = {};
            auto load_scales = [&](int u) {
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const int row = min(nb + rank * p.R + ((w_in_set + 4 * e) >> 1) * 32 + lane, p.n_pad - 1);   // (rows past the matrix are never stored)
                    const float* s = p.scale_grp + ((size_t)(row >> 7) * p.units + u) * 256 + (row & 127);
                    sc_next[e][0] = __ldg(s);
                    sc_next[e][1] = __ldg(s + 128);
                }
            };
            if constexpr (MODE == W_U4C) load_scales(u0);
            int slot = 0, rslot = 0, turn = 0;
            // A part is folded, where the ring of widened slabs holds a piece, when one has been widened behind it: the MMAs of the
            // next part wait for the fold, and go on at once with the slabs that are there.
            constexpr int BEHIND = SPU <= SETS ? 1 : 0;
            int fold_at = parts > 1 ? part_unit(1) + BEHIND : n_units;
            unsigned phase = 0, rphase = 0;
            for (int j = 0; j < n_units && ok; j++) {
                const int u = u0 + j;
                if constexpr (FOLD) {
                    if (j == fold_at) {
                        fold_part();
                        if (!ok) break;
                        fold_at = folds < parts - 1 ? part_unit(folds + 1) + BEHIND : n_units;
                    }
                }
                if constexpr (MODE == W_U4C) {
#pragma unroll
                    for (int e = 0; e < 4; e++) { sc[e][0] = sc_next[e][0]; sc[e][1] = sc_next[e][1]; }
                    if (j + 1 < n_units) load_scales(u0 + j + 1);
                }
                ok = __all_sync(0xffffffffu, mbar_wait(bar_raw_full + 8 * rslot, rphase, abort_flag, p.wait_limit_ns));
                if (!ok) break;
                const unsigned char* raw = raw_ring + rslot * w_bytes;
                // (not unrolled: the warps are at different places of this code, and four copies of it outgrow the
                // instruction cache)
#pragma unroll 1
                for (int s = 0; s < SPU; s++) {
                    if (u * SPU + s >= p.slabs) break;          // warp-uniform: the last piece may reach past K
                    if (turn == set) {
                        constexpr int UNITS = MODE == W_U8C ? 2 : 1;     // 16-byte units of an item's row
                        uint4 v[4][UNITS];
#pragma unroll
                        for (int e = 0; e < 4; e++) {
                            const int item = w_in_set + 4 * e, row = (item >> 1) * 32 + lane, kh = item & 1;
                            if (item >= n_items) break;
                            // 4 bits: the unit that holds K [64 s + 32 kh, +32) of the piece (see quant4_kernel in pack.cu)
#pragma unroll
                            for (int q = 0; q < UNITS; q++)
                                v[e][q] = *(const uint4*)(raw + row * SLAB_BYTES +
                                                          (((MODE == W_U8C ? 4 * s + 2 * kh + q : 4 * (s & 1) + 2 * kh + (s >> 1)) ^ (row & 7)) << 4));
                        }
                        ok = __all_sync(0xffffffffu, mbar_wait(bar_wide_empty + 8 * slot, phase ^ 1, abort_flag, p.wait_limit_ns));
                        if (!ok) break;
                        unsigned char* dst = wide_ring + slot * w_bytes;
#pragma unroll
                        for (int e = 0; e < 4; e++) {
                            const int item = w_in_set + 4 * e, row = (item >> 1) * 32 + lane, kh = item & 1, sw = row & 7;
                            if (item >= n_items) break;
                            unsigned char* d = dst + row * SLAB_BYTES;
                            if constexpr (MODE == W_U8C) {
#pragma unroll
                                for (int q = 0; q < 2; q++) {
                                    const uint4 b = v[e][q];
                                    *(uint4*)(d + (((4 * kh + 2 * q) ^ sw) << 4)) =
                                        make_uint4(u8x2_to_bf16x2(b.x, 0x4140), u8x2_to_bf16x2(b.x, 0x4342),
                                                   u8x2_to_bf16x2(b.y, 0x4140), u8x2_to_bf16x2(b.y, 0x4342));
                                    *(uint4*)(d + (((4 * kh + 2 * q + 1) ^ sw) << 4)) =
                                        make_uint4(u8x2_to_bf16x2(b.z, 0x4140), u8x2_to_bf16x2(b.z, 0x4342),
                                                   u8x2_to_bf16x2(b.w, 0x4140), u8x2_to_bf16x2(b.w, 0x4342));
                                }
                            } else {
                                const unsigned w4[4] = {v[e][0].x, v[e][0].y, v[e][0].z, v[e][0].w};
                                const float f = s < 2 ? sc[e][0] : sc[e][1];
#pragma unroll
                                for (int q = 0; q < 4; q++)
                                    *(uint4*)(d + (((4 * kh + q) ^ sw) << 4)) =
                                        make_uint4(nib2_to_bf16x2_scaled(w4[q], f), nib2_to_bf16x2_scaled(w4[q] >> 4, f),
                                                   nib2_to_bf16x2_scaled(w4[q] >> 8, f), nib2_to_bf16x2_scaled(w4[q] >> 12, f));
                            }
                        }
                        // the widened bytes must be visible to the tensor core (async proxy) before the slot counts as full
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                        __syncwarp();
                        if (lane == 0) {
                            if (CG == 1 || leader) mbar_arrive(bar_wide_full + 8 * slot);
                            else mbar_arrive_leader(leader_full + 8 * slot);
                        }
                    }
                    if (++turn == SETS) turn = 0;
                    if (++slot == p.wide_slots) { slot = 0; phase ^= 1; }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_raw_empty + 8 * rslot);
                if (++rslot == p.raw_slots) { rslot = 0; rphase ^= 1; }
            }
        }
        if constexpr (FOLD)
            while (folds < parts - 1 && ok) fold_part();        // (a part shorter than the ring)
        // ---------------- epilogue ----------------
        asm volatile("bar.sync 1, %0;" ::"n"(WORKERS * 32) : "memory");
        ok = __all_sync(0xffffffffu, ok && mbar_wait<32>(bar_acc, 0, abort_flag, p.wait_limit_ns));
        tc_fence_after();
        const int m = (tm * CG + rank) * BM + quarter * 32 + lane;
        const bool row_ok = m < p.M;
        // accumulator column of a chunk -> output column: with a pair, MMA 0 holds the first R0 columns of CTA 0's R and of
        // CTA 1's R side by side, MMA 1 the other R - R0 of both
        auto chunk_col = [&](int c) -> int {
            if constexpr (CG == 1) return c * 32;
            const int h = c * 32 >= 2 * p.R0, rows = h ? p.R - p.R0 : p.R0, cc = c * 32 - (h ? 2 * p.R0 : 0);
            const int r = cc >= rows;
            return r * p.R + (h ? p.R0 : 0) + cc - (r ? rows : 0);
        };
        // columns [32 c, +32) of this CTA's result: the sums of the folded parts, if any, and the last part's accumulators in order
        const int filled = min(p.sets, n_slabs - part_slab(parts - 1));
        auto load_acc = [&](int c, unsigned (&r)[32]) {
            if (FOLD && parts > 1) {
                load_sums(c, r);
            } else {
                tc_ld32(taddr + (unsigned)(c * 32), r);
                tc_wait_ld();
            }
            if constexpr (!I8) {
#pragma unroll 1
                for (int t = parts > 1 ? 0 : 1; t < filled; t++) {
                    unsigned x[32];
                    tc_ld32(taddr + (unsigned)(t * W + c * 32), x);
                    tc_wait_ld();
#pragma unroll
                    for (int j = 0; j < 32; j++) r[j] = __float_as_uint(__uint_as_float(r[j]) + __uint_as_float(x[j]));
                }
            }
        };
        if (p.S > 1) {
            // Part `q` of K hands chunk c of its accumulators to CTA (c mod S) of the cluster: 16 KB at slot (c / S) * S + q of
            // that CTA's ring, as [4-column piece][row] 16-byte units.  Remote stores are posted, so nothing waits for a
            // round trip (reading the other CTAs' sums took 3 us per chunk); the ring has to be free in every CTA first.
            const unsigned mine = smem_u32(smem) + (unsigned)((quarter * 32 + lane) * 16);
            __syncwarp();
            cluster_sync_all();
            if (ok) {
#pragma unroll 1
                for (int c = third; c < chunks; c += SETS) {
                    unsigned r[32];
                    load_acc(c, r);
                    const int owner = c % p.S;
                    const unsigned dst = mapa_rank(mine + (unsigned)(((c / p.S) * p.S + split) * CHUNK_BYTES), (unsigned)(owner * CG + rank));
#pragma unroll
                    for (int j = 0; j < 8; j++)
                        st_cluster_v4(dst + (unsigned)(j * BM * 16), r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
                }
            }
            __syncwarp();
            cluster_sync_all();
        }
        // accumulators of the t-th chunk this CTA finishes: its own, or the sum of the parts in the order of K
        auto fetch = [&](int t, int c, unsigned (&r)[32]) {
            if (p.S == 1) {
                load_acc(c, r);
                return;
            }
            const uint4* src = (const uint4*)(smem + t * p.S * CHUNK_BYTES) + quarter * 32 + lane;
#pragma unroll
            for (int j = 0; j < 32; j++) r[j] = 0;      // (0 + x = x, and a part of -0 ends as +0 like any sum with it)
#pragma unroll 2
            for (int q = 0; q < p.S; q++) {
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const uint4 v = src[q * (CHUNK_BYTES / 16) + j * BM];
                    const unsigned x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        if (I8) r[4 * j + e] += x[e];
                        else r[4 * j + e] = __float_as_uint(__uint_as_float(r[4 * j + e]) + __uint_as_float(x[e]));
                    }
                }
            }
        };
        // every load of the ring has landed and every MMA has read it: the staging tiles lie at its end
        EpiArgs ea{p.ep, p.vec_ok, I8 ? 1 : 0, p.n1, p.M, (unsigned*)(smem + RING_BYTES - (WORKERS - wi) * WARP_TILE_BYTES)};
        auto set_vecs = [&](int col) {
            if (use_deq) ea.cv_deq = colvec + col;
            if (use_bias) ea.cv_bias = colvec + MAX_W + col;
            if (use_q) ea.cv_q = colvec + 2 * MAX_W + col;
        };
        const int kind = epilogue_kind(p.ep, p.vec_ok);
        if (ok) {
            for_epilogue_kind<MODE == W_I8_HALF>(kind, I8, [&](auto k) {
#pragma unroll 1
                for (int t = third, c = split + third * p.S; c < chunks; t += SETS, c += SETS * p.S) {
                    const int col = chunk_col(c);
                    if (nb + col + 32 > p.n1) continue;      // (warp-uniform)
                    unsigned r[32];
                    fetch(t, c, r);
                    set_vecs(col);
                    epilogue_whole<decltype(k)::value>(r, m, nb + col, ea);
                }
            });
#pragma unroll 1
            for (int t = third, c = split + third * p.S; c < chunks; t += SETS, c += SETS * p.S) {
                const int col = chunk_col(c);
                if (nb + col >= p.n1 || (kind != EPI_GENERAL && nb + col + 32 <= p.n1)) continue;
                unsigned r[32];
                fetch(t, c, r);
                set_vecs(col);
                epilogue_chunk(r, m, nb + col, ea, row_ok);
            }
        }
        __syncwarp();
    }
    if (warp < 4 && p.S > 1) {
        __syncwarp();
        cluster_sync_all();   // (the workers' barriers around the exchange of partial sums)
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
        if constexpr (CG == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
    }
}

// ---- host side ----------------------------------------------------------------------------------------------------------
struct WaveShape { int cg, R, S, tiles_m, tiles_n; };

template <int CG, int MODE, bool FOLD>
int allow_smem() {
    static std::atomic<unsigned long long> attr_devices{0};
    return once_per_device(attr_devices, [] {
        B200FC_CUDA(cudaFuncSetAttribute(gemm_wave_kernel<CG, MODE, FOLD>, cudaFuncAttributeMaxDynamicSharedMemorySize, WAVE_SMEM));
        return (int)B200FC_OK;
    });
}

template <int CG>
int max_tiles(int S, int* out) {
    static ClusterCounts counts;
    int n = 0;
    const int rc = resident_clusters(counts, CG * S, WAVE_THREADS, WAVE_SMEM, &n);
    if (rc) return rc;
    const int by_sms = num_sms() / (CG * S);
    *out = n < by_sms ? n : by_sms;
    return B200FC_OK;
}

int max_sets(int W) { return 512 / W < 8 ? 512 / W : 8; }   // accumulators of W columns in tensor memory
// parts that `chains` chains of sums in a CTA take
int parts_of(int chains, int W) { return (chains + max_sets(W) - 1) / max_sets(W); }

// Picks the columns per CTA and the split of K of a call that fits one wave; false = it does not.  The model counts SM
// clocks of one CTA: per 128-byte slab the slowest of operand loads (about 48 bytes per clock and SM reach shared memory from
// L2), MMAs (the 256-wide one takes 128 clocks per 32 bytes of K) and widening; plus the reduction and the epilogue.
// `chains`: the number of chains that K is to be summed in at least, see k_chains.
template <int CG, int MODE>
int pick_shape(int M, int nspan, int slabs, int units, int chains, WaveShape* best, bool* found) {
    const int tiles_m = (M + BM * CG - 1) / (BM * CG);
    const int rows_a = M < BM ? M : BM;
    const int wbytes = MODE == W_U4C ? 34 : (MODE == W_U8C ? 64 : 128);
    double best_cost = 0;
    *found = false;
    for (int S = 1; S * CG <= 8 && S <= units; S++) {
        int cap = 0;
        const int rc = max_tiles<CG>(S, &cap);
        if (rc) return rc;
        for (int R = 32; R <= 256; R += 32) {
            const int W = R * CG, tiles_n = (nspan + W - 1) / W;
            if ((long long)tiles_m * tiles_n > cap) continue;
            const int parts = parts_of((chains + S - 1) / S, W);
            if (parts > 1 && MODE != W_U8C && MODE != W_U4C) continue;    // (plain weights never need it: their chains are fewer)
            if (S > 1 && S * ((W / 32 + S - 1) / S) * CHUNK_BYTES + WORKERS * WARP_TILE_BYTES > RING_BYTES) continue;
            const double load = (rows_a * 128.0 + R * (double)wbytes) / 48.0, mma = 2.0 * W;
            const double cvt = MODE == W_U4C ? 2.2 * R : (MODE == W_U8C ? 1.4 * R : 0.0);
            double slab = load > mma ? load : mma;
            if (cvt > slab) slab = cvt;
            const double hbm = (double)nspan * slabs * wbytes / 3400.0;
            double loop = slab * ((slabs + S - 1) / S);
            if (loop < hbm) loop = hbm;
            const double red = S > 1 ? 1500.0 + W * 4.0 + W * 512.0 * (S - 1) / S / 30.0 : 0.0;
            const double fold = (parts - 1) * (600.0 + 4.0 * W);
            const double cost = loop + red + fold + 400.0 * ((W / 32 + 2 * S - 1) / (2 * S));
            if (!*found || cost < best_cost) {
                *found = true;
                best_cost = cost;
                *best = WaveShape{CG, R, S, tiles_m, tiles_n};
            }
        }
    }
    return B200FC_OK;
}

struct WaveCall {
    const Weight& w;
    const void* A;
    int M, K;
    int64_t lda;
    bool a_signed;
    const Epilogue& ep;
    cudaStream_t s;
    int slabs, units, chains;
};

template <int CG, int MODE>
int run_wave(const WaveCall& call, const WaveShape& sh, int n0, int n1) {
    constexpr bool I8 = MODE == W_I8 || MODE == W_I8_HALF, WQ = MODE == W_U8C || MODE == W_U4C;
    constexpr int SPU = MODE == W_U8C ? 2 : (MODE == W_U4C ? 4 : 1);
    const Epilogue& ep = call.ep;
    const int64_t w_ld = call.w.ld_bytes();
    const bool w_signed = call.w.dtype == B200FC_S8;
    WaveParams p = {};
    p.slabs = call.slabs; p.units = call.units;
    p.M = call.M; p.n0 = n0; p.n1 = n1; p.n_pad = call.w.N_pad;
    p.R = sh.R; p.S = sh.S; p.tiles_m = sh.tiles_m;
    const int chains = (call.chains + sh.S - 1) / sh.S;
    p.parts = parts_of(chains, CG * sh.R);
    p.sets = (chains + p.parts - 1) / p.parts;
    const int grid = CG * sh.S * sh.tiles_m * sh.tiles_n;
    bool own_sums = false;
    if (p.parts > 1) {
        // the workspace of the split of K in gemm_tc.cu, which this takes the place of; memory of the graph where the stream is being captured
        int rc = get_stream_scratch((size_t)grid * (CG * sh.R / 32) * CHUNK_BYTES, call.s, 1, (void**)&p.sums, &own_sums);
        if (rc) return rc;
    }
    p.R0 = CG == 2 && sh.R > 128 ? (sh.R / 2 + 31) / 32 * 32 : sh.R;
    p.idesc0 = make_idesc(I8, call.a_signed, w_signed, CG * p.R0, CG * BM);
    p.idesc1 = make_idesc(I8, call.a_signed, w_signed, CG * (p.R - p.R0), CG * BM);
    const int a_bytes = BM * SLAB_BYTES, w_bytes = sh.R * SLAB_BYTES;
    if (WQ) {
        // three widened slabs (more measured no faster); stored pieces for six slabs and more ahead (HBM latency); the rest
        // for activations
        p.wide_slots = 3;
        p.slots = sh.R <= 192 ? 4 : 3;
        p.raw_slots = (RING_BYTES - p.wide_slots * w_bytes - p.slots * a_bytes) / w_bytes;
        if (p.raw_slots > (SPU == 4 ? 3 : 5)) p.raw_slots = SPU == 4 ? 3 : 5;
        p.slots = (RING_BYTES - (p.wide_slots + p.raw_slots) * w_bytes) / a_bytes;
    } else {
        p.slots = RING_BYTES / (a_bytes + w_bytes);
    }
    if (p.slots > MAX_SLOTS) p.slots = MAX_SLOTS;
    p.ep = ep;
    p.scale_grp = call.w.scale_grp;
    p.status = kernel_status_word();
    if (!p.status) { set_error("gemm: no kernel status word on this device"); return B200FC_ERR_CUDA; }
    p.wait_limit_ns = wait_limit_ns();
    p.vec_ok = output_vec(ep, n0, I8);

    CUtensorMap ma, mw;
    int rc = make_map(&ma, call.A, I8, (uint64_t)call.K, (uint64_t)call.M, (uint64_t)call.lda, BM);
    if (rc) return rc;
    rc = WQ ? make_map(&mw, call.w.data, true, (uint64_t)w_ld, (uint64_t)call.w.N_pad, (uint64_t)w_ld, (uint32_t)p.R)
            : make_map(&mw, call.w.data, I8, (uint64_t)call.w.K_pad, (uint64_t)call.w.N_pad, (uint64_t)w_ld, (uint32_t)p.R);
    if (rc) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid, 1, 1);
    cfg.blockDim = dim3(WAVE_THREADS, 1, 1);
    cfg.dynamicSmemBytes = WAVE_SMEM;
    cfg.stream = call.s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)(CG * sh.S);
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    if (p.parts == 1) {
        rc = allow_smem<CG, MODE, false>();
        if (rc) return rc;
        B200FC_CUDA(cudaLaunchKernelEx(&cfg, gemm_wave_kernel<CG, MODE, false>, ma, mw, p));
    } else if constexpr (WQ) {
        rc = allow_smem<CG, MODE, true>();
        if (rc) return rc;
        B200FC_CUDA(cudaLaunchKernelEx(&cfg, gemm_wave_kernel<CG, MODE, true>, ma, mw, p));
        if (own_sums) B200FC_CUDA(cudaFreeAsync(p.sums, call.s));
    }
    count_launch();
    const int tile[6] = {CG, p.R, p.S, p.sets, p.parts, sh.tiles_m * sh.tiles_n};
    for (int i = 0; i < 6; i++) last_wave_tile()[i] = tile[i];
    return B200FC_OK;
}

// The tensor core's error grows with the length of a chain of fp32 sums (256 x 4096 x 4096, relative to float64: 1.08e-6 in three
// chains, 7.9e-7 in four, 5.1e-7 in six).  K is cut into at least as many chains as launch_gemm_tc cuts it into.  For quantised weights
// that is a number for each block of rows that would be widened in front of it (fewer columns, more parts): the error
// of the whole result, as the root mean square of 1 / chains, must not be larger.
int k_chains(const Weight& w, int M, int K, int n0, int n1) {
    if (!w.compressed) return gemm_tc_chains(M, K, n1 - n0);
    const int blk = widened_block_rows(w.K_pad);
    double sum = 0.0;
    for (int r0 = n0 / kRowPad * kRowPad; r0 < n1; r0 += blk) {
        const int cols = (r0 + blk < n1 ? r0 + blk : n1) - (r0 > n0 ? r0 : n0), c = gemm_tc_chains(M, K, cols);
        sum += (double)cols / (c * c);
    }
    int chains = 1;
    while ((double)(n1 - n0) / (chains * chains) > sum * 1.000001) chains++;
    return chains;
}

// Calls with quantised weights that do not fit one wave and are faster through blocks of widened weights than in gemm_qt.cu: many rows
// and short K.  Widening costs what K x N does, once; the epilogue of gemm_qt, longer per element than that of gemm_tc, and its
// conversion per tile grow with the rows.  The line is drawn through 245 timed calls of 600 to 4096 rows, K 1024 to 4096, N 3072 to 21248: it loses
// 0.4 % on average and 11 % at most against the faster of the two (us, blocks / gemm_qt: int8 4096 x 1024 x 11008 86 / 115,
// 3000 x 1408 x 21248 144 / 159, 1400 x 1408 x 11008 50.3 / 50.6, 3000 x 2304 x 6016 68.7 / 67.7, 2000 x 1792 x 21248 149 / 124; 4 bits
// 4096 x 1024 x 11008 81 / 123, 2000 x 1408 x 6016 42.9 / 47.2, 3000 x 2304 x 11008 137 / 125; with GeLU int8 3000 x 1408 x 11008 91 / 117).
// Fewer than 400 rows are not widened for, however short K: 300 x 128 x 40000 37 / 33, 100 x 64 x 40000 33 / 14, 400 x 256 x 40000 41 / 48.
// A capturing stream stays with gemm_qt, which needs no workspace.
bool faster_in_blocks(const WaveCall& c, bool w4, int nspan) {
    const bool one_block = nspan <= widened_block_rows(c.w.K_pad);
    if (c.M < 400 || c.M < (one_block ? 1.25 : 1.9) * c.K * (w4 ? 0.75 : 1.0) * (c.ep.steps & B200FC_STEP_GELU ? 0.8 : 1.0)) return false;
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    return cudaStreamIsCapturing(c.s, &st) == cudaSuccess && st == cudaStreamCaptureStatusNone;
}

template <int MODE>
int run_wave(WaveCall& c, int n0, int n1) {
    constexpr bool WQ = MODE == W_U8C || MODE == W_U4C;
    constexpr int SPU = MODE == W_U8C ? 2 : (MODE == W_U4C ? 4 : 1);
    const int slab_elems = MODE == W_I8 || MODE == W_I8_HALF ? SLAB_BYTES : SLAB_BYTES / 2;
    c.slabs = (c.K + slab_elems - 1) / slab_elems;
    c.units = MODE == W_U4C ? (int)(c.w.ld_bytes() / SLAB_BYTES) : (c.slabs + SPU - 1) / SPU;     // (the group scales are laid out by it)
    WaveShape sh;
    bool found = false;
    const int rc = c.M <= BM ? pick_shape<1, MODE>(c.M, n1 - n0, c.slabs, c.units, c.chains, &sh, &found)
                             : pick_shape<2, MODE>(c.M, n1 - n0, c.slabs, c.units, c.chains, &sh, &found);
    if (rc) return rc;
    if constexpr (WQ) {
        // Quantised weights: gemm_qt.cu takes most calls that do not fit one wave (us, through blocks of widened weights / there: int8
        // 571 x 10624 x 21504 575 / 201, 1071 x 2560 x 22784 210 / 112, 4096 x 4096 x 11008 289 / 239; 4 bits 3526 x 8448 x 10168
        // 575 / 449), and of the others those of up to 512 rows and those whose K would be split (us, here / there: int8 22 x 3840 x 6016
        // 26.4 / 11.8, 158 x 3840 x 8576 37.0 / 26.5, 949 x 8704 x 2048 39.8 / 34.3; 4 bits 33 x 2400 x 9824 21.7 / 14.6).  More rows in tiles
        // of all of K are level or faster here, whatever the post-ops (bias, bf16 / bias, GeLU, bf16 / plain fp32, here : there: int8
        // 705 x 2560 x 10240 34.4 : 35.0 / 39.4 : 40.7 / 35.8 : 34.5, 2017 x 1408 x 4200 27.5 : 29.8 / 33.2 : 35.7 / 29.1 : 28.8; 4 bits
        // 705 x 2560 x 10240 38.7 : 43.6 / 43.5 : 47.6 / 39.4 : 42.9; not all: int8 1689 x 1920 x 1920 20.5 : 18.7 / 22.7 : 20.8 / 21.1 : 18.5).
        // 4 bits with more than 64 rows and many chains are nearly level (100 x 4096 x 11008 26.4 : 25.6 / 27.5 : 26.9 / 26.6 : 25.6).  Folded calls would be faster there as
        // well (4 bits 300 x 4096 x 11008 59.5 / 40.4), but their tiles are what b200fc_last_wave_tile reports and stay.  K is summed in
        // no fewer chains than it would be here.
        // fp32 behind GeLU (sums_pinned): only where K is one chain on either path, which gives the same bits (slabs < 96: a ragged last
        // round of blocks of widened weights is split along K from there on).
        const bool pinned = MODE == W_U8C && sums_pinned(c.ep);
        if (!found && (!pinned || (c.chains == 1 && c.slabs < 96)) && !faster_in_blocks(c, MODE == W_U4C, n1 - n0))
            return launch_gemm_qt(c.w, c.A, c.M, c.K, c.lda, n0, n1, c.ep, c.chains, false, c.s);
        if (found && !pinned) {
            const int W = sh.cg * sh.R, chains = (c.chains + sh.S - 1) / sh.S, parts = parts_of(chains, W);
            const bool level = MODE == W_U4C && c.M > 64 && sh.S * chains > 4;
            if (parts == 1 && !level && (c.M <= 512 || sh.S > 1))
                return launch_gemm_qt(c.w, c.A, c.M, c.K, c.lda, n0, n1, c.ep, sh.S * chains, true, c.s);
        }
    }
    if (!found) return B200FC_ERR_UNSUPPORTED;
    // 256 x 256 tiles without a split of K are gemm_tc.cu's own, whose loop is a little better (us, here / there: 150 x 6272 x 14256
    // 46.8 / 42.7, 250 x 2784 x 14928 27.6 / 26.7)
    if (!WQ && sh.cg == 2 && sh.S == 1 && sh.R == 128 && 4 * sh.tiles_m * sh.tiles_n > num_sms()) return B200FC_ERR_UNSUPPORTED;
    return sh.cg == 1 ? run_wave<1, MODE>(c, sh, n0, n1) : run_wave<2, MODE>(c, sh, n0, n1);
}

}  // namespace

int* last_wave_tile() {
    static thread_local int tile[6];
    return tile;
}

int launch_gemm_wave(const Weight& w, const void* A, int dtypeA, int M, int K, int64_t lda, int n0, int n1, const Epilogue& ep,
                     cudaStream_t s) {
    if (M <= 0 || n1 <= n0) return B200FC_OK;
    if (ep.mc_reduce || (((uintptr_t)A | (uintptr_t)lda) & 15)) return B200FC_ERR_UNSUPPORTED;
    static int enabled = -1;                       // B200FC_GEMM_WAVE=0, or a GEMM forced by its own switch: never
    if (enabled < 0) { const char* e = getenv("B200FC_GEMM_WAVE"); enabled = (e ? atoi(e) : 1) && !gemm_forced_ctas(); }
    if (!enabled) return B200FC_ERR_UNSUPPORTED;
    const bool a8 = dtypeA != B200FC_BF16;
    WaveCall c{w, A, M, K, lda, dtypeA == B200FC_S8, ep, s, 0, 0, a8 ? 1 : k_chains(w, M, K, n0, n1)};   // (sums of 8-bit products are exact)
    if (w.compressed) return w.dtype == B200FC_S4 ? run_wave<W_U4C>(c, n0, n1) : run_wave<W_U8C>(c, n0, n1);
    if (a8) return output_vec(ep, n0, true) == 2 ? run_wave<W_I8_HALF>(c, n0, n1) : run_wave<W_I8>(c, n0, n1);
    return run_wave<W_BF16>(c, n0, n1);
}

}  // namespace b200fc
