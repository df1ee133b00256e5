// Decode-shaped fully-connected layer (M <= 16 rows of bf16 activations) with quantised weights, on the tensor cores.
//
// Replaces the M <= 16 branches of the compressed-weight specialisation Matmul<bf16,int8_t,float>
// (include/kernels_amx.hpp:1381-1441) for int8 and 4-bit weights; gemv_tma.cu keeps bf16 weights and unaligned activations.
//
// The stream of weights is that of gemv_tma.cu: stages of 128 rows x 128 bytes by TMA, S CTAs (one cluster) per row block of 128
// whose partial sums meet in distributed shared memory.  What differs is the product: with mma.sync it took 28 clocks of an SM
// quarter per 16 x 8 x 16 step, more than the stream itself from 8 rows on.  Here eight warps widen the weights to bf16 in
// registers and put them into tensor memory, one row per TMEM lane, as the A operand of tcgen05.mma; the activations
// ([16 rows] x 64 K tiles that travel with the stage) are the B operand.  Widened weights never touch shared memory, whose
// bandwidth they would exceed (five bytes per weight instead of two), activations are not converted, and sixteen rows cost
// what one costs.
// Both kinds are widened to 64ths of their values, which are exact in bf16, with one fused multiply-add per pair: with four instructions
// per pair of int8 weights instead of two 16 x 4096 x 11008 took 14.5 us, not 12.7, and 4 bits 4 x 4096 x 11008 11.9, not 11.1.
//   int8   : exact in bf16; the stages take four fp32 accumulators (or eight) in turn, which are added at the end: the tensor core's error
//            grows with the length of a chain of sums (16 x 4096 x 11008, relative to float64: 1.9e-7 in one chain, 0.8e-7 in
//            four, 1.1e-7 with mma.sync's chains).
//   4 bits : the integers are multiplied; every group of 128 K has an accumulator of its own, which the warp of its rows reads
//            back and adds, times the group's fp32 scale, to sums in registers.
// Warps: 0 = TMA producer, 1 = MMA issuer and TMEM owner, 2-3 idle, 4-11 = widening in two sets of four (one warp per TMEM
// quarter) that take the pieces of 128 rows x 128 K in turn; the sets' warps then finish the row block.
// Barriers: full / empty per ring stage, a_full / a_empty per A buffer in tensor memory, d_full / d_empty per group accumulator.
// Every wait is bounded as in gemm_tc.cu.
#include <cstdlib>
#include "tc_common.cuh"

namespace b200fc {

namespace {

constexpr int TQ_ROWS = 128;
constexpr int TQ_THREADS = 384;
constexpr int A_COLS = 64, D_COLS = 16;           // an A buffer: 128 K of bf16; an accumulator: 16 rows of activations
constexpr int TQ_TMEM = 256;                      // two CTAs share an SM's 512 columns
constexpr int X_TILE = 16 * SLAB_BYTES;           // 16 rows x 64 K of activations
constexpr int W_STAGE = TQ_ROWS * SLAB_BYTES;

// LONG: for calls whose K is split less than the places for CTAs would allow, so that the chains of sums get no longer.  int8: two A
// buffers and eight accumulators instead of three and four (4 x 4096 x 5032: 10.4 us, 10.2 without).  4 bits: a second level of
// sums in registers (4 x 4096 x 11008, which is not such a call: 12.5 us, 11.8 without).
template <int WB, bool LONG = false> struct TqLayout {
    static constexpr int PIECES = WB == 4 ? 2 : 1;                    // pieces of 128 K per stage
    static constexpr int STAGES = WB == 4 ? 4 : 5;
    static constexpr int A_BUFS = LONG && WB == 8 ? 2 : 3, D_BUFS = (TQ_TMEM - A_BUFS * A_COLS) / D_COLS;
    static constexpr int X_BYTES = PIECES * 2 * X_TILE;
    static constexpr int SC_BYTES = WB == 4 ? 2 * TQ_ROWS * 4 : 0;    // the stage's 2 x 128 group scales
    static constexpr int STAGE = W_STAGE + X_BYTES + SC_BYTES;
    static constexpr int PART_OFF = STAGES * STAGE;                   // [16 rows][128 columns] fp32
    static constexpr int EP_OFF = PART_OFF + 16 * TQ_ROWS * 4;
    static constexpr int BAR_OFF = EP_OFF + 3 * TQ_ROWS * 4;
    static constexpr int SMEM = BAR_OFF + 256 + 1024;
};

struct TqParams {
    int spr, S;               // stages per packed row; CTAs per row block
    int M, n0, n1;
    Epilogue ep;
    const float* scales;      // 4-bit weights: [row block][stage][2][128]
    int* status;
    unsigned long long wait_limit_ns;
};

template <int WB, bool LONG>
__global__ void __launch_bounds__(TQ_THREADS, 2)
gemv_tq_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const TqParams p) {
    using L = TqLayout<WB, LONG>;
    constexpr int PIECES = L::PIECES, STAGES = L::STAGES, A_BUFS = L::A_BUFS, D_BUFS = L::D_BUFS;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = smem_raw + (((smem_u32(smem_raw) + 1023u) & ~1023u) - smem_u32(smem_raw));
    float* part = (float*)(smem + L::PART_OFF);
    float* s_ep = (float*)(smem + L::EP_OFF);
    const unsigned bar_full = smem_u32(smem + L::BAR_OFF), bar_empty = bar_full + 8 * STAGES;
    const unsigned bar_a_full = bar_empty + 8 * STAGES, bar_a_empty = bar_a_full + 8 * A_BUFS;
    const unsigned bar_d_full = bar_a_empty + 8 * A_BUFS, bar_d_empty = bar_d_full + 8 * D_BUFS;   // int8: d_full[0] = all done
    unsigned* tmem_holder = (unsigned*)(smem + L::BAR_OFF + 8 * (2 * STAGES + 2 * A_BUFS + 2 * D_BUFS));
    volatile int* abort_flag = (volatile int*)(tmem_holder + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rb = (int)blockIdx.x / p.S, rank = (int)blockIdx.x % p.S;
    const int row0 = p.n0 + rb * TQ_ROWS;
    const int st0 = (int)((long long)p.spr * rank / p.S), n_st = (int)((long long)p.spr * (rank + 1) / p.S) - st0;
    const int n_pieces = n_st * PIECES;
    const unsigned long long limit = p.wait_limit_ns;

    if (threadIdx.x == 0) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_x) : "memory");
        for (int i = 0; i < STAGES; i++) { mbar_init(bar_full + 8 * i, 1); mbar_init(bar_empty + 8 * i, 1); }
        for (int i = 0; i < A_BUFS; i++) { mbar_init(bar_a_full + 8 * i, 4); mbar_init(bar_a_empty + 8 * i, 1); }
        for (int i = 0; i < D_BUFS; i++) { mbar_init(bar_d_full + 8 * i, 1); mbar_init(bar_d_empty + 8 * i, 4); }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (warp == 0) {
        // ---------------- producer: the first ring of weights travels before anything else ----------------
        auto load_w = [&](int i, int slot) {
            const unsigned dst = smem_u32(smem + slot * L::STAGE), full = bar_full + 8 * slot;
            mbar_expect_tx(full, L::STAGE);
            tma_load_2d(dst, &map_w, full, (st0 + i) * SLAB_BYTES, row0);
            if constexpr (WB == 4)
                bulk_load_1d(dst + W_STAGE + L::X_BYTES, p.scales + ((size_t)(row0 / TQ_ROWS) * p.spr + st0 + i) * (2 * TQ_ROWS),
                             L::SC_BYTES, full);
        };
        auto load_x = [&](int i, int slot) {
            const unsigned dst = smem_u32(smem + slot * L::STAGE) + W_STAGE, full = bar_full + 8 * slot;
#pragma unroll
            for (int t = 0; t < 2 * PIECES; t++) tma_load_2d(dst + t * X_TILE, &map_x, full, ((st0 + i) * 2 * PIECES + t) * 64, 0);
        };
        const int pre = min(STAGES, n_st);
        for (int i = 0; i < pre; i++)
            if (elect_one()) load_w(i, i);
        asm volatile("griddepcontrol.wait;" ::: "memory");
        for (int i = 0; i < pre; i++)
            if (elect_one()) load_x(i, i);
        int slot = 0;
        unsigned phase = 0;          // (every slot is used for the second time from here on)
        for (int i = pre; i < n_st; i++) {
            if (!__all_sync(0xffffffffu, mbar_wait(bar_empty + 8 * slot, phase, abort_flag, limit))) break;
            if (elect_one()) { load_w(i, slot); load_x(i, slot); }
            if (++slot == STAGES) { slot = 0; phase ^= 1; }
        }
    } else if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_holder)), "r"((unsigned)TQ_TMEM) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (warp != 0) {
        // everyone but the producer: the tensor memory is there
        tc_fence_before();
        asm volatile("bar.sync 2, %0;" ::"n"(TQ_THREADS - 32) : "memory");
        tc_fence_after();
    }
    // the next kernel of the stream may become resident (not earlier: it could take the tensor memory this CTA still needs)
    if (warp == 1) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const unsigned tmem_base = warp != 0 ? *(volatile unsigned*)tmem_holder : 0;
    const unsigned tmem_d = tmem_base + A_BUFS * A_COLS;

    if (warp == 1) {
        // ---------------- MMA issue ----------------
        const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((16u >> 3) << 17) | ((128u >> 4) << 24);   // bf16 x bf16 -> fp32, N 16, M 128
        int slot = 0, ab = 0, db = 0;
        unsigned phase = 0, a_phase = 0, d_phase = 0;
        bool ok = true;
        for (int i = 0; i < n_st && ok; i++) {
            ok = __all_sync(0xffffffffu, mbar_wait(bar_full + 8 * slot, phase, abort_flag, limit));
#pragma unroll
            for (int h = 0; h < PIECES; h++) {
                if (ok) ok = __all_sync(0xffffffffu, mbar_wait(bar_a_full + 8 * ab, a_phase, abort_flag, limit));
                if (WB == 4 && ok) ok = __all_sync(0xffffffffu, mbar_wait(bar_d_empty + 8 * db, d_phase ^ 1, abort_flag, limit));
                if (!ok) break;
                tc_fence_after();
                const unsigned long long bdesc = make_smem_desc(smem_u32(smem + slot * L::STAGE) + W_STAGE + h * 2 * X_TILE);
                if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < 8; k++)
                        tc_mma_ts(tmem_d + (WB == 4 ? db : i % D_BUFS) * D_COLS, tmem_base + ab * A_COLS + k * 8,
                                  bdesc + (unsigned long long)((k >> 2) * (X_TILE >> 4) + (k & 3) * (MMA_K_BYTES >> 4)), idesc,
                                  (unsigned)(WB == 4 ? k != 0 : (i >= D_BUFS || k != 0)));
                    tc_commit(bar_a_empty + 8 * ab);
                    if (WB == 4) tc_commit(bar_d_full + 8 * db);
                    if (h == PIECES - 1) {
                        tc_commit(bar_empty + 8 * slot);
                        if (WB != 4 && i == n_st - 1) tc_commit(bar_d_full);
                    }
                }
                if (++ab == A_BUFS) { ab = 0; a_phase ^= 1; }
                if (WB == 4 && ++db == D_BUFS) { db = 0; d_phase ^= 1; }
            }
            if (++slot == STAGES) { slot = 0; phase ^= 1; }
        }
        __syncwarp();
    } else if (warp >= 4) {
        // ---------------- widening ----------------
        const int set = (warp - 4) >> 2, quarter = warp & 3, row = quarter * 32 + lane, sw = row & 7;
        const unsigned lane_base = (unsigned)(quarter * 32) << 16;
        const Epilogue& ep = p.ep;
        bool ok = true;
        float acc[16], total[16];       // (total: 4 bits and LONG, the sums of eight groups of a set)
#pragma unroll
        for (int t = 0; t < 16; t++) acc[t] = total[t] = 0.0f;
        float sc_prev = 0.0f;
        // 4 bits: group sum of piece g -> acc += sum * scale
        auto take_group = [&](int g, float sc) {
            const int db = g % D_BUFS;
            ok = __all_sync(0xffffffffu, mbar_wait(bar_d_full + 8 * db, (unsigned)(g / D_BUFS) & 1, abort_flag, limit));
            if (!ok) return;
            tc_fence_after();
            unsigned r[16];
            tc_ld16(tmem_d + lane_base + db * D_COLS, r);
            tc_wait_ld();
#pragma unroll
            for (int t = 0; t < 16; t++) acc[t] = fmaf(__uint_as_float(r[t]), sc, acc[t]);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_d_empty + 8 * db);
            if (LONG && ((g >> 1) & 7) == 7) {
#pragma unroll
                for (int t = 0; t < 16; t++) { total[t] += acc[t]; acc[t] = 0.0f; }
            }
        };
#pragma unroll 1
        for (int g = set; g < n_pieces && ok; g += 2) {
            const int i = g / PIECES, slot = i % STAGES, ab = g % A_BUFS;
            ok = __all_sync(0xffffffffu, mbar_wait(bar_full + 8 * slot, (unsigned)(i / STAGES) & 1, abort_flag, limit));
            if (!ok) break;
            const unsigned char* src = smem + slot * L::STAGE + row * SLAB_BYTES;
            float sc = 0.0f;
            if constexpr (WB == 4) sc = ((const float*)(smem + slot * L::STAGE + W_STAGE + L::X_BYTES))[set * TQ_ROWS + row];
#pragma unroll
            for (int h = 0; h < 2; h++) {              // 64 K each: 32 columns of tensor memory
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
                    // units of group `set`: K [32 j, +32) of the group in unit 2 j + set (see quant4_kernel in pack.cu)
#pragma unroll
                    for (int u = 0; u < 2; u++) {
                        const uint4 v = *(const uint4*)(src + (((2 * (2 * h + u) + set) ^ sw) << 4));
                        const unsigned w4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                        for (int q = 0; q < 4; q++) nib8_to_bf16x2_64th(w4[q], &r[16 * u + 4 * q]);
                    }
                }
                if (h == 0) {
                    ok = __all_sync(0xffffffffu, mbar_wait(bar_a_empty + 8 * ab, ((unsigned)(g / A_BUFS) & 1) ^ 1, abort_flag, limit));
                    if (!ok) break;
                    tc_fence_after();
                }
                tc_st32(tmem_base + lane_base + ab * A_COLS + h * 32, r);
            }
            if (!ok) break;
            tc_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_a_full + 8 * ab);
            if constexpr (WB == 4) {
                if (g >= 2) take_group(g - 2, sc_prev);
                sc_prev = sc;
            }
        }
        // per-row vectors of the post-ops (the previous kernel of the stream may have written them)
        asm volatile("griddepcontrol.wait;" ::: "memory");
        if (set == 1) {
            const int n = row0 + row;
            float deq = 1.0f, bias = 0.0f, q = 1.0f;
            if (n < p.n1) {
                if (ep.steps & B200FC_STEP_DEQUANT) deq = ep.deq_per_oc ? ep.deq_scale * ep.deq_per_oc[n] : ep.deq_scale;
                if (ep.steps & B200FC_STEP_BIAS) bias = ep.bias[n];
                if (ep.steps & B200FC_STEP_QUANT) q = ep.q_per_oc ? ep.q_per_oc[n] : ep.q_scale;
            }
            s_ep[row] = deq; s_ep[TQ_ROWS + row] = bias; s_ep[2 * TQ_ROWS + row] = q;
        }
        if constexpr (WB == 4) {
            const int last = n_pieces - 2 + set;       // (a set's last piece; n_pieces is even)
            if (ok && last >= 0) take_group(last, sc_prev);
            if constexpr (LONG) {
#pragma unroll
                for (int t = 0; t < 16; t++) acc[t] += total[t];
            }
        } else if (set == 0) {
            ok = __all_sync(0xffffffffu, ok && mbar_wait(bar_d_full, 0, abort_flag, limit));
            tc_fence_after();
            for (int d = 0; d < min(D_BUFS, n_st); d++) {
                unsigned r[16];
                tc_ld16(tmem_d + lane_base + d * D_COLS, r);
                tc_wait_ld();
#pragma unroll
                for (int t = 0; t < 16; t++) acc[t] += __uint_as_float(r[t]);
            }
        }
        if (set == 0) {
#pragma unroll
            for (int t = 0; t < 16; t++)
                if (t < p.M) part[t * TQ_ROWS + row] = acc[t] * 64.0f;          // (the weights are in 64ths)
        }
        if constexpr (WB == 4) {      // the two sets' sums: even groups plus odd groups
            asm volatile("bar.sync 1, 256;" ::: "memory");
            if (set == 1) {
#pragma unroll
                for (int t = 0; t < 16; t++)
                    if (t < p.M) part[t * TQ_ROWS + row] += acc[t] * 64.0f;
            }
        }
        __syncwarp();
    }
    __syncwarp();

    // ---- the S parts of the row block meet: every CTA of the cluster finishes 1/S of the outputs, adding in rank order ----
    tc_fence_before();
    if (p.S > 1) cluster_sync_all();
    else __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((unsigned)TQ_TMEM) : "memory");
    }
    if (!*abort_flag) {
        const Epilogue& ep = p.ep;
        const unsigned part_addr = smem_u32(part);
        const int n_out = TQ_ROWS * p.M;
        const int e0 = (int)((long long)n_out * rank / p.S), e1 = (int)((long long)n_out * (rank + 1) / p.S);
        // (the previous kernel of the stream may still read what this one overwrites; warps 1-3 have not waited for it yet)
        asm volatile("griddepcontrol.wait;" ::: "memory");
        for (int e = e0 + (int)threadIdx.x; e < e1; e += TQ_THREADS) {
            const int tok = e / TQ_ROWS, row = e % TQ_ROWS, n = row0 + row;
            const float sum = cluster_sum(part_addr + 4u * (unsigned)e, p.S);
            if (n >= p.n1) continue;
            float v = sum;
            if (ep.steps & B200FC_STEP_DEQUANT) v *= s_ep[row];
            if (ep.steps & B200FC_STEP_BIAS) v += s_ep[TQ_ROWS + row];
            if (ep.steps & B200FC_STEP_GELU) v = gelu_erf_poly(v);
            if (ep.steps & B200FC_STEP_QUANT) v *= s_ep[2 * TQ_ROWS + row];
            store_scalar(v, tok, n, ep);
        }
    } else if (threadIdx.x == 0) {
        atomicExch(p.status, 3);
        const unsigned long long t0 = globaltimer();
        while (globaltimer() - t0 < 200000ull) { }   // copies still in flight land before shared memory is released
    }
    __syncwarp();
    if (p.S > 1) cluster_sync_all();   // nobody leaves while a peer may still read its partial sums
    else __syncthreads();
}

template <int WB, bool LONG>
int run_tq(const CUtensorMap& mw, const CUtensorMap& mx, const TqParams& p, int grid, cudaStream_t s) {
    using L = TqLayout<WB, LONG>;
    static std::atomic<unsigned long long> attr_devices{0};
    const int arc = once_per_device(attr_devices, [] {
        B200FC_CUDA(cudaFuncSetAttribute(gemv_tq_kernel<WB, LONG>, cudaFuncAttributeMaxDynamicSharedMemorySize, L::SMEM));
        return (int)B200FC_OK;
    });
    if (arc) return arc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid, 1, 1);
    cfg.blockDim = dim3(TQ_THREADS, 1, 1);
    cfg.dynamicSmemBytes = L::SMEM;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)p.S;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    B200FC_CUDA(cudaLaunchKernelEx(&cfg, gemv_tq_kernel<WB, LONG>, mw, mx, p));
    count_launch();
    return B200FC_OK;
}

}  // namespace

// max_ctas: CTAs that may be resident at once (two per SM unless the caller has been given fewer)
int launch_gemv_tq(const Weight& w, const void* A, int M, int K, int64_t lda, int n0, int n1, const Epilogue& ep, int max_ctas,
                   cudaStream_t s) {
    const int es = w.dtype == B200FC_S4 ? 4 : (w.dtype == B200FC_S8 && w.compressed ? 8 : 0);
    if (!es || M < 1 || M > 16 || (((uintptr_t)A | (uintptr_t)lda) & 15) || (ep.steps & B200FC_STEP_SILU_MUL)) return B200FC_ERR_UNSUPPORTED;
    if (es == 4 && (!w.scale_grp || (n0 % TQ_ROWS))) return B200FC_ERR_UNSUPPORTED;
    TqParams p = {};
    p.spr = (int)(w.ld_bytes() / SLAB_BYTES);
    const int row_blocks = (n1 - n0 + TQ_ROWS - 1) / TQ_ROWS;
    // More row blocks than half of the places for CTAs (max_ctas): K is not split (S = 1 below) and the places beyond the row blocks
    // stay empty.  With long rows that imbalance costs more than the faster product gains, and gemv_tma.cu cuts the stream into equal
    // pieces (us, there / here: int8 1 x 8192 x 20480 36.9 / 47.0, x 28672 46.0 / 47.7; 4 bits 8 x 8192 x 25088 35.6 / 40.6;
    // 16 rows int8 x 20480 45.4 / 48.6, x 25088 51.5 / 49.4; K = 3328 is level at 1 row and 1.2 to 1.3 times faster here at 16).  The
    // same with one place per SM, where the line lies at 74 row blocks: int8 1 x 4096 x 10240 22.7 / 24.7, x 12800 25.3 / 25.1,
    // 1 x 8192 x 12800 38.5 / 46.2; 16 rows 4096 x 12800 33.8 / 27.3.  (Row blocks that fill all places would be faster here: 1 x 4096 x 18944
    // 24.2 / 18.1.)  The lines between are drawn through these sizes.
    if (2 * row_blocks > max_ctas && (M <= 8 ? K >= 4096 : K >= 8192 && 7 * row_blocks < 4 * max_ctas)) return B200FC_ERR_UNSUPPORTED;
    // as many parts of K per row block as keep all CTAs resident, of two stages and more each
    int S = max_ctas / row_blocks;
    if (S > 8) S = 8;
    if (S > p.spr / 2) S = p.spr / 2;
    if (S < 1) S = 1;
    const int places_S = S;
    static ClusterCounts counts;
    int rc = sums_pinned(ep) ? B200FC_OK       // (two CTAs per SM with either layout)
                             : fit_clusters(counts, TQ_THREADS, es == 4 ? TqLayout<4>::SMEM : TqLayout<8>::SMEM, row_blocks, &S);
    if (rc) return rc;
    p.S = S;
    p.M = M; p.n0 = n0; p.n1 = n1;
    p.ep = ep;
    p.scales = w.scale_grp;
    p.status = kernel_status_word();
    if (!p.status) { set_error("gemv: no kernel status word on this device"); return B200FC_ERR_CUDA; }
    p.wait_limit_ns = wait_limit_ns();
    CUtensorMap mw, mx;
    rc = make_map(&mw, w.data, true, (uint64_t)w.ld_bytes(), (uint64_t)w.N_pad, (uint64_t)w.ld_bytes(), TQ_ROWS);
    if (rc) return rc;
    rc = make_map(&mx, A, false, (uint64_t)K, (uint64_t)M, (uint64_t)lda, 16);
    if (rc) return rc;
    const int grid = row_blocks * S;
    if (S < places_S) return es == 4 ? run_tq<4, true>(mw, mx, p, grid, s) : run_tq<8, true>(mw, mx, p, grid, s);
    return es == 4 ? run_tq<4, false>(mw, mx, p, grid, s) : run_tq<8, false>(mw, mx, p, grid, s);
}

}  // namespace b200fc
