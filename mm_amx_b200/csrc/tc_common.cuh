// What the tcgen05 GEMM kernels share: PTX wrappers, operand and instruction descriptors, tensor maps, and the epilogue on a
// 32-column chunk of one output row.
#pragma once
#include <cuda.h>
#include "common.cuh"

namespace b200fc {

namespace {

constexpr int BM = 128;
constexpr int SLAB_BYTES = 128;          // K extent of one pipeline stage, in bytes of operand elements
constexpr int MMA_K_BYTES = 32;          // K extent of one tcgen05.mma (16 bf16 / 32 int8)

#ifndef B200FC_EPI_SLEEP_NS
#define B200FC_EPI_SLEEP_NS 256
#endif
constexpr int EPI_SLEEP_NS = B200FC_EPI_SLEEP_NS;

// staging tile of an epilogue warp: 32 rows x 32 four-byte columns, or (HALF below) 32 x 16, which four-byte outputs go through twice
constexpr int EPI_TILE_WORDS = 32 * 32;

// ---- PTX wrappers ------------------------------------------------------------------------------------------------
__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned long long globaltimer() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ void mbar_init(unsigned bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// CLUSTER: acquires at cluster scope, for a phase that arrivals of another CTA of the cluster complete
template <bool CLUSTER = false>
__device__ __forceinline__ bool mbar_try_wait(unsigned bar, unsigned parity) {
    unsigned ok;
    if constexpr (CLUSTER) {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
    } else {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
    }
    return ok != 0;
}
// Bounded wait.  Returns false when the CTA is aborting (this wait or another role's ran out of time).
// The clock and the abort flag are looked at after a batch of failed attempts only (try_wait itself suspends the thread for a while).
// SLEEP_NS > 0: back off between polls (for waits that are long and not latency critical: the epilogue warps wait most
// of a tile's main loop, and five spinning warps cost issue slots and power that the tensor pipe could use).
template <int SLEEP_NS = 0, bool CLUSTER = false>
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity, volatile int* abort_flag, unsigned long long limit) {
    if (mbar_try_wait<CLUSTER>(bar, parity)) return true;
    unsigned long long t0 = 0;
    while (true) {
#pragma unroll 1
        for (int i = 0; i < 16; i++) {
            if (SLEEP_NS > 0) __nanosleep(SLEEP_NS);
            if (mbar_try_wait<CLUSTER>(bar, parity)) return true;
        }
        if (*abort_flag) return false;
        const unsigned long long now = globaltimer();
        if (t0 == 0) t0 = now;
        if (now - t0 > limit) {
            *abort_flag = 1;
            return false;
        }
    }
}
__device__ __forceinline__ void tma_load_2d(unsigned dst, const CUtensorMap* map, unsigned bar, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y)
        : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(unsigned bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
template <bool I8>
__device__ __forceinline__ void tc_mma(unsigned d_tmem, unsigned long long adesc, unsigned long long bdesc,
                                       unsigned idesc, unsigned accumulate) {
    if constexpr (I8) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
            : "memory");
    } else {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
            : "memory");
    }
}
__device__ __forceinline__ void tc_ld32(unsigned taddr, unsigned (&r)[32]) {
    __syncwarp();      // (lanes of rows past M may have left the previous chunk early; the load is a warp-wide instruction)
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ void tc_st32(unsigned taddr, const unsigned (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
          "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]),
          "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]),
          "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// D (128 rows) += A (128 x 16, tensor memory) x B (columns x 16, shared memory)
__device__ __forceinline__ void tc_mma_ts(unsigned d_tmem, unsigned a_tmem, unsigned long long bdesc, unsigned idesc, unsigned accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// Shared-memory operand descriptor: K-major tile, rows of 128 bytes, 128-byte swizzle, 8-row groups 1024 bytes
// apart (stride-dimension byte offset); descriptor version 1 (Blackwell).
__device__ __forceinline__ unsigned long long make_smem_desc(unsigned smem_addr) {
    unsigned long long d = 0;
    d |= (unsigned long long)((smem_addr & 0x3FFFFu) >> 4);
    d |= (unsigned long long)1 << 16;            // leading-dimension byte offset (unused for swizzled K-major)
    d |= (unsigned long long)(1024 >> 4) << 32;  // stride-dimension byte offset
    d |= (unsigned long long)1 << 46;            // descriptor version
    d |= (unsigned long long)2 << 61;            // SWIZZLE_128B
    return d;
}

// ---- epilogue on 32 consecutive columns of one output row ------------------------------------------------------------
struct EpiArgs {       // what the epilogue of one 32-column chunk needs to know
    Epilogue ep;       // (by value: the fields then live in registers)
    int vec_ok, acc_is_int, n1;    // (vec_ok: see output_vec)
    int M;             // rows of the output
    unsigned* tile;    // this warp's staging tile in shared memory (EPI_TILE_WORDS words)
    // the chunk's 32 per-column values, staged in shared memory ahead of the tile (16-byte aligned), or null: read
    // them from global memory
    const float* cv_deq = nullptr;
    const float* cv_bias = nullptr;
    const float* cv_q = nullptr;
};
// Output rows leave through shared memory: the lanes of a warp hold one row each, and their direct stores would write 32
// scattered pieces of 16 bytes.  A warp's staging tile keeps UNITS 16-byte units per row (8: 32 four-byte values; 4: 32 bf16;
// 2: 32 int8 or 16 bf16); unit j of row r sits at position j ^ swizzle(r), so that neither pass has bank conflicts.
template <int UNITS>
__device__ __forceinline__ int tile_pos(int row, int unit) {
    return row * UNITS + (unit ^ (UNITS == 8 ? (row & 7) : (UNITS == 4 ? ((row >> 1) & 3) : ((row >> 2) & 1))));
}
// the tile -> rows [m0, m0 + 32) of C, byte columns [c0, c0 + 16 UNITS): every store instruction writes whole row segments
template <int UNITS>
__device__ __forceinline__ void flush_tile(const unsigned* tile, char* C, long long ldc, int m0, long long c0, int M) {
    constexpr int ROWS = 32 / UNITS;                 // rows per store instruction
    const int lane = threadIdx.x & 31, unit = lane % UNITS;
    __syncwarp();
    char* dst = C + (long long)(m0 + lane / UNITS) * ldc + c0 + unit * 16;
#pragma unroll
    for (int it = 0; it < UNITS; it++) {
        const int row = it * ROWS + lane / UNITS;
        const uint4 q = ((const uint4*)tile)[tile_pos<UNITS>(row, unit)];
        if (m0 + row < M) *(uint4*)(dst + (long long)(it * ROWS) * ldc) = q;
    }
    __syncwarp();
}
// the same for int8 rows that are only 8-byte aligned (UNITS = 2): four lanes per row segment of 32 bytes
__device__ __forceinline__ void flush_tile_s8_half(const unsigned* tile, char* C, long long ldc, int m0, long long c0, int M) {
    const int lane = threadIdx.x & 31, half = lane & 3;
    __syncwarp();
    char* dst = C + (long long)(m0 + (lane >> 2)) * ldc + c0 + half * 8;
#pragma unroll
    for (int it = 0; it < 4; it++) {
        const int row = it * 8 + (lane >> 2);
        const uint2 q = ((const uint2*)tile)[2 * tile_pos<2>(row, half >> 1) + (half & 1)];
        if (m0 + row < M) *(uint2*)(dst + (long long)(it * 8) * ldc) = q;
    }
    __syncwarp();
}
// two fp32 values in a 64-bit register: one instruction of sm_100a works on both, rounding each like the scalar form
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// gelu_erf_poly (common.cuh) on eight values: the same operations in the same order for each, four chains of pairs side by side
__device__ __forceinline__ void gelu_erf_poly8(f32x2 (&v)[4]) {
    constexpr unsigned coef[15] = {0x1f1c83fdu, 0xa3198977u, 0x268a7927u, 0xa998c963u, 0x2c67ddb2u, 0xaf013b2cu, 0x315d4a4fu,
                                   0xb3969b11u, 0x35a776e9u, 0xb79b0914u, 0x3970b255u, 0xbb1b7399u, 0x3ca3621fu, 0xbe082bc7u,
                                   0x3f4c4228u};
    f32x2 x2[4], q[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        x2[j] = mul2(v[j], v[j]);
        q[j] = pack2(__uint_as_float(coef[0]), __uint_as_float(coef[0]));
    }
#pragma unroll
    for (int i = 1; i < 15; i++) {
        const f32x2 c = pack2(__uint_as_float(coef[i]), __uint_as_float(coef[i]));
#pragma unroll
        for (int j = 0; j < 4; j++) q[j] = fma2(q[j], x2[j], c);
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const f32x2 xh = mul2(v[j], pack2(0.5f, 0.5f));
        float x[2], h[2], y[2];
        unpack2(v[j], x[0], x[1]);
        unpack2(xh, h[0], h[1]);
        unpack2(mul2(fma2(q[j], v[j], pack2(1.0f, 1.0f)), xh), y[0], y[1]);
#pragma unroll
        for (int e = 0; e < 2; e++) {
            float far;      // x < -5 -> 0, x > 5 -> x, NaN -> NaN
            asm("max.NaN.f32 %0, %1, 0f00000000;" : "=f"(far) : "f"(x[e]));
            const float ax = fabsf(x[e]);
            if (!(ax <= 5.0f)) y[e] = far;
            if (ax <= __uint_as_float(0x33800000u)) y[e] = h[e];
        }
        v[j] = pack2(y[0], y[1]);
    }
}
// four fp32 -> four int8, as f32_to_s8 (round to nearest even, saturate, NaN -> -128) but off the conversion unit, whose 16
// values per clock and SM bound an int8 epilogue: clamp, then the rounding of adding 1.5 * 2^23 leaves the integer in the
// low byte
__device__ __forceinline__ unsigned f32x4_to_s8x4(float a, float b, float c, float d) {
    const float magic = 12582912.0f;
    const unsigned ua = __float_as_uint(fminf(fmaxf(a, -128.0f), 127.0f) + magic), ub = __float_as_uint(fminf(fmaxf(b, -128.0f), 127.0f) + magic);
    const unsigned uc = __float_as_uint(fminf(fmaxf(c, -128.0f), 127.0f) + magic), ud = __float_as_uint(fminf(fmaxf(d, -128.0f), 127.0f) + magic);
    return __byte_perm(__byte_perm(ua, ub, 0x0040), __byte_perm(uc, ud, 0x0040), 0x5410);
}
// the per-column values vec[n .. n + 8) (every lane needs all of them): from the copy staged for the chunk, as two 16-byte loads
// where they are whole and aligned, else as scalar loads clamped to the last valid column
__device__ __forceinline__ void load_col_vec(const float* staged, const float* __restrict__ vec, int n, int n1, f32x2 (&out)[4]) {
    float4 t[2];
    if (staged) {
        t[0] = ((const float4*)staged)[0];
        t[1] = ((const float4*)staged)[1];
    } else if (n + 8 <= n1 && (((uintptr_t)(vec + n)) & 15) == 0) {
        t[0] = __ldg((const float4*)(vec + n));
        t[1] = __ldg((const float4*)(vec + n) + 1);
    } else {
        float* f = (float*)t;
#pragma unroll
        for (int j = 0; j < 8; j++) f[j] = __ldg(vec + min(n + j, n1 - 1));
    }
#pragma unroll
    for (int h = 0; h < 2; h++) { out[2 * h] = pack2(t[h].x, t[h].y); out[2 * h + 1] = pack2(t[h].z, t[h].w); }
}
__device__ __forceinline__ unsigned pack_bf16x2(float lo, float hi) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *(const unsigned*)&h;
}
// Post-ops and store of 32 consecutive columns [n, n + 32) of one output row per lane, whose accumulators are in `acc`.  Called by
// all lanes of the warp.  This is the form for everything: chunks at the ragged end, unaligned outputs, residuals, multicast.
template <bool HALF = false>
__device__ __forceinline__ void epilogue_chunk(const unsigned (&acc)[32], int m, int n, const EpiArgs& p, bool row_ok, long long c_offset = 0) {
    const Epilogue& ep = p.ep;
    const bool staged = p.vec_ok && (!p.acc_is_int || p.vec_ok == 1) && n + 32 <= p.n1 && !ep.mc_reduce;   // warp-uniform
    const int lane = threadIdx.x & 31, m0 = m - lane;
    char* Cb = (char*)ep.C + c_offset;
    char* crow = Cb + (long long)m * ep.ldc;
    uint4* tile = (uint4*)p.tile;

    if (ep.steps & B200FC_STEP_SILU_MUL) {
        // columns [0,16) gate, [16,32) up of the same 16 channels -> 16 bf16 outputs at column n / 2
        if (!row_ok) return;
        unsigned short* dst = (unsigned short*)crow + (n >> 1);
#pragma unroll
        for (int j = 0; j < 16; j++)
            if (n + 16 + j < p.n1) dst[j] = f32_to_bf16_bits(silu_f(__uint_as_float(acc[j])) * __uint_as_float(acc[16 + j]));
        return;
    }

#pragma unroll
    for (int q = 0; q < 4; q++) {
        unsigned r[8];
#pragma unroll
        for (int j = 0; j < 8; j++) r[j] = acc[8 * q + j];
        const int nq = n + 8 * q;
        if (ep.out_dtype != B200FC_S32) {
            f32x2 w[4];
#pragma unroll
            for (int j = 0; j < 4; j++)
                w[j] = p.acc_is_int ? pack2((float)(int)r[2 * j], (float)(int)r[2 * j + 1])
                                    : pack2(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1]));
            f32x2 cv[4];
            if (ep.steps & B200FC_STEP_DEQUANT) {
                const f32x2 one = pack2(ep.deq_scale, ep.deq_scale);
                if (ep.deq_per_oc) load_col_vec(p.cv_deq ? p.cv_deq + 8 * q : nullptr, ep.deq_per_oc, nq, p.n1, cv);
#pragma unroll
                for (int j = 0; j < 4; j++) w[j] = mul2(w[j], ep.deq_per_oc ? mul2(one, cv[j]) : one);
            }
            if (ep.steps & B200FC_STEP_BIAS) {
                load_col_vec(p.cv_bias ? p.cv_bias + 8 * q : nullptr, ep.bias, nq, p.n1, cv);
#pragma unroll
                for (int j = 0; j < 4; j++) w[j] = add2(w[j], cv[j]);
            }
            if (ep.steps & B200FC_STEP_GELU) gelu_erf_poly8(w);
            if (ep.steps & B200FC_STEP_QUANT) {
                const f32x2 one = pack2(ep.q_scale, ep.q_scale);
                if (ep.q_per_oc) load_col_vec(p.cv_q ? p.cv_q + 8 * q : nullptr, ep.q_per_oc, nq, p.n1, cv);
#pragma unroll
                for (int j = 0; j < 4; j++) w[j] = mul2(w[j], ep.q_per_oc ? cv[j] : one);
            }
            float v[8];
#pragma unroll
            for (int j = 0; j < 4; j++) unpack2(w[j], v[2 * j], v[2 * j + 1]);
            if (ep.residual && row_ok) {
                // residual added in fp32, before the one rounding of the output
                const char* rrow = (const char*)ep.residual + (long long)m * ep.ld_res;
                if (staged && (((uintptr_t)rrow + (size_t)nq * 2) & 15) == 0) {
                    const int4 t = __ldg((const int4*)(rrow + (long long)nq * 2));
                    const unsigned w4[4] = {(unsigned)t.x, (unsigned)t.y, (unsigned)t.z, (unsigned)t.w};
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        v[2 * e] += __uint_as_float(w4[e] << 16);
                        v[2 * e + 1] += __uint_as_float(w4[e] & 0xffff0000u);
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < 8; j++)
                        v[j] += __uint_as_float((unsigned)((const unsigned short*)rrow)[min(nq + j, p.n1 - 1)] << 16);
                }
            }
#pragma unroll
            for (int j = 0; j < 8; j++) r[j] = __float_as_uint(v[j]);
        }
        auto f = [&](int j) { return __uint_as_float(r[j]); };
        if (staged) {
            if (ep.out_dtype == B200FC_BF16) {
                tile[tile_pos<4>(lane, q)] = make_uint4(pack_bf16x2(f(0), f(1)), pack_bf16x2(f(2), f(3)), pack_bf16x2(f(4), f(5)), pack_bf16x2(f(6), f(7)));
            } else if (ep.out_dtype == B200FC_S8) {
                ((uint2*)tile)[2 * tile_pos<2>(lane, q >> 1) + (q & 1)] = make_uint2(f32x4_to_s8x4(f(0), f(1), f(2), f(3)), f32x4_to_s8x4(f(4), f(5), f(6), f(7)));
            } else if constexpr (HALF) {
                tile[tile_pos<4>(lane, 2 * (q & 1))] = make_uint4(r[0], r[1], r[2], r[3]);
                tile[tile_pos<4>(lane, 2 * (q & 1) + 1)] = make_uint4(r[4], r[5], r[6], r[7]);
                if (q & 1) flush_tile<4>(p.tile, Cb, ep.ldc, m0, (long long)(n + 16 * (q >> 1)) * 4, p.M);
            } else {
                tile[tile_pos<8>(lane, 2 * q)] = make_uint4(r[0], r[1], r[2], r[3]);
                tile[tile_pos<8>(lane, 2 * q + 1)] = make_uint4(r[4], r[5], r[6], r[7]);
            }
        } else if (!row_ok) {
        } else if (ep.mc_reduce) {
            // Fused all-reduce: C is a multicast mapping of the output on every GPU of the tensor-parallel group; the NVSwitch
            // adds this rank's contribution into all replicas (multimem.red), so no separate collective runs.
            const bool full = p.vec_ok && n + 32 <= p.n1;
            if (ep.out_dtype == B200FC_F32) {
                float* dst = (float*)(crow + (long long)nq * 4);
                if (full) {
#pragma unroll
                    for (int j = 0; j < 2; j++)
                        asm volatile("multimem.red.relaxed.sys.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst + 4 * j),
                                     "f"(f(4 * j)), "f"(f(4 * j + 1)), "f"(f(4 * j + 2)), "f"(f(4 * j + 3))
                                     : "memory");
                } else {
#pragma unroll
                    for (int j = 0; j < 8; j++)
                        if (nq + j < p.n1) asm volatile("multimem.red.relaxed.sys.global.add.f32 [%0], %1;" ::"l"(dst + j), "f"(f(j)) : "memory");
                }
            } else {
                unsigned short* dst = (unsigned short*)(crow + (long long)nq * 2);
                const unsigned o[4] = {pack_bf16x2(f(0), f(1)), pack_bf16x2(f(2), f(3)), pack_bf16x2(f(4), f(5)), pack_bf16x2(f(6), f(7))};
                if (full) {
                    asm volatile("multimem.red.relaxed.sys.global.add.v4.bf16x2 [%0], {%1, %2, %3, %4};" ::"l"(dst), "r"(o[0]), "r"(o[1]),
                                 "r"(o[2]), "r"(o[3])
                                 : "memory");
                } else {
#pragma unroll
                    for (int j = 0; j < 4; j++)   // the launcher guarantees an even column range for this mode
                        if (nq + 2 * j + 1 < p.n1)
                            asm volatile("multimem.red.relaxed.sys.global.add.bf16x2 [%0], %1;" ::"l"(dst + 2 * j), "r"(o[j]) : "memory");
                }
            }
        } else {
#pragma unroll
            for (int j = 0; j < 8; j++) {
                if (nq + j >= p.n1) break;
                if (ep.out_dtype == B200FC_BF16) ((unsigned short*)crow)[nq + j] = f32_to_bf16_bits(f(j));
                else if (ep.out_dtype == B200FC_S8) ((signed char*)crow)[nq + j] = (signed char)f32_to_s8(f(j));
                else ((unsigned*)crow)[nq + j] = r[j];
            }
        }
    }
    if (staged) {
        if (ep.out_dtype == B200FC_BF16) flush_tile<4>(p.tile, Cb, ep.ldc, m0, (long long)n * 2, p.M);
        else if (ep.out_dtype == B200FC_S8) flush_tile<2>(p.tile, Cb, ep.ldc, m0, n, p.M);
        else if constexpr (!HALF) flush_tile<8>(p.tile, Cb, ep.ldc, m0, (long long)n * 4, p.M);
    }
}
// 32 four-byte columns of a row per lane through the staging tile
template <bool HALF>
__device__ __forceinline__ void store_words(const unsigned (&v)[32], unsigned* staging, char* C, long long ldc, int m0, int n, int M) {
    uint4* tile = (uint4*)staging;
    const int lane = threadIdx.x & 31;
    constexpr int UNITS = HALF ? 4 : 8;
#pragma unroll
    for (int h = 0; h < 8 / UNITS; h++) {
#pragma unroll
        for (int j = 0; j < UNITS; j++) {
            const int i = 4 * (h * UNITS + j);
            tile[tile_pos<UNITS>(lane, j)] = make_uint4(v[i], v[i + 1], v[i + 2], v[i + 3]);
        }
        flush_tile<UNITS>(staging, C, ldc, m0, (long long)(n + 16 * h) * 4, M);
    }
}
// The same for whole aligned chunks without residual and multicast, i.e. nearly all of them: one output kind per
// instantiation, and one branch per post-op and chunk.  (With the choice made inside, per eight columns, a chunk took 2400
// clocks of a warp for a plain bf16 store.)
template <int V> struct IntConst { static constexpr int value = V; };
enum EpiKind { EPI_F32 = 0, EPI_BF16, EPI_S8, EPI_S32, EPI_SILU, EPI_S8_HALF, EPI_GENERAL };
__device__ __forceinline__ int epilogue_kind(const Epilogue& ep, int vec_ok) {
    if (!vec_ok || ep.mc_reduce || ep.residual) return EPI_GENERAL;
    if (vec_ok == 2) return EPI_S8_HALF;
    if (ep.steps & B200FC_STEP_SILU_MUL) return EPI_SILU;
    return ep.out_dtype == B200FC_F32 ? EPI_F32 : (ep.out_dtype == B200FC_BF16 ? EPI_BF16 : (ep.out_dtype == B200FC_S8 ? EPI_S8 : EPI_S32));
}
template <int KIND, bool HALF = false>
__device__ __forceinline__ void epilogue_whole(const unsigned (&acc)[32], int m, int n, const EpiArgs& p, long long c_offset = 0) {
    const Epilogue& ep = p.ep;
    const int lane = threadIdx.x & 31, m0 = m - lane;
    char* C = (char*)ep.C + c_offset;
    uint4* tile = (uint4*)p.tile;
    if constexpr (KIND == EPI_SILU) {
        // A lane's 16 values are one 32-byte sector: stored directly, the way through shared memory only adds latency.  Rows past M
        // stay out of the arithmetic as well: their accumulators are zeros, and a division of zero takes the slow path of
        // the division (94 us instead of 58 for 436 x 3072 x 20096).
        if (m < p.M) {
            float y[16];
#pragma unroll
            for (int j = 0; j < 16; j++) y[j] = silu_f(__uint_as_float(acc[j])) * __uint_as_float(acc[16 + j]);
            uint4* dst = (uint4*)(C + (long long)m * ep.ldc + n);       // column n / 2, two bytes each
#pragma unroll
            for (int h = 0; h < 2; h++)
                dst[h] = make_uint4(pack_bf16x2(y[8 * h], y[8 * h + 1]), pack_bf16x2(y[8 * h + 2], y[8 * h + 3]),
                                    pack_bf16x2(y[8 * h + 4], y[8 * h + 5]), pack_bf16x2(y[8 * h + 6], y[8 * h + 7]));
        }
        __syncwarp();
        return;
    } else if constexpr (KIND == EPI_S32) {
        store_words<HALF>(acc, p.tile, C, ep.ldc, m0, n, p.M);
        return;
    } else {
        f32x2 w[16];
#pragma unroll
        for (int j = 0; j < 16; j++)
            w[j] = p.acc_is_int ? pack2((float)(int)acc[2 * j], (float)(int)acc[2 * j + 1])
                                : pack2(__uint_as_float(acc[2 * j]), __uint_as_float(acc[2 * j + 1]));
        if (ep.steps & B200FC_STEP_DEQUANT) {
            const f32x2 one = pack2(ep.deq_scale, ep.deq_scale);
            if (ep.deq_per_oc) {
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    f32x2 cv[4];
                    load_col_vec(p.cv_deq ? p.cv_deq + 8 * q : nullptr, ep.deq_per_oc, n + 8 * q, p.n1, cv);
#pragma unroll
                    for (int j = 0; j < 4; j++) w[4 * q + j] = mul2(w[4 * q + j], mul2(one, cv[j]));
                }
            } else {
#pragma unroll
                for (int j = 0; j < 16; j++) w[j] = mul2(w[j], one);
            }
        }
        if (ep.steps & B200FC_STEP_BIAS) {
#pragma unroll
            for (int q = 0; q < 4; q++) {
                f32x2 cv[4];
                load_col_vec(p.cv_bias ? p.cv_bias + 8 * q : nullptr, ep.bias, n + 8 * q, p.n1, cv);
#pragma unroll
                for (int j = 0; j < 4; j++) w[4 * q + j] = add2(w[4 * q + j], cv[j]);
            }
        }
        if (ep.steps & B200FC_STEP_GELU) {
#pragma unroll
            for (int q = 0; q < 4; q++) {
                f32x2 t[4] = {w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]};
                gelu_erf_poly8(t);
#pragma unroll
                for (int j = 0; j < 4; j++) w[4 * q + j] = t[j];
            }
        }
        if (ep.steps & B200FC_STEP_QUANT) {
            const f32x2 one = pack2(ep.q_scale, ep.q_scale);
            if (ep.q_per_oc) {
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    f32x2 cv[4];
                    load_col_vec(p.cv_q ? p.cv_q + 8 * q : nullptr, ep.q_per_oc, n + 8 * q, p.n1, cv);
#pragma unroll
                    for (int j = 0; j < 4; j++) w[4 * q + j] = mul2(w[4 * q + j], cv[j]);
                }
            } else {
#pragma unroll
                for (int j = 0; j < 16; j++) w[j] = mul2(w[j], one);
            }
        }
        float v[32];
#pragma unroll
        for (int j = 0; j < 16; j++) unpack2(w[j], v[2 * j], v[2 * j + 1]);
        if constexpr (KIND == EPI_F32) {
            unsigned o[32];
#pragma unroll
            for (int j = 0; j < 32; j++) o[j] = __float_as_uint(v[j]);
            store_words<HALF>(o, p.tile, C, ep.ldc, m0, n, p.M);
        } else if constexpr (KIND == EPI_BF16) {
#pragma unroll
            for (int j = 0; j < 4; j++)
                tile[tile_pos<4>(lane, j)] = make_uint4(pack_bf16x2(v[8 * j], v[8 * j + 1]), pack_bf16x2(v[8 * j + 2], v[8 * j + 3]),
                                                        pack_bf16x2(v[8 * j + 4], v[8 * j + 5]), pack_bf16x2(v[8 * j + 6], v[8 * j + 7]));
            flush_tile<4>(p.tile, C, ep.ldc, m0, (long long)n * 2, p.M);
        } else {
            unsigned o[8];
#pragma unroll
            for (int j = 0; j < 8; j++) o[j] = f32x4_to_s8x4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
#pragma unroll
            for (int h = 0; h < 2; h++) tile[tile_pos<2>(lane, h)] = make_uint4(o[4 * h], o[4 * h + 1], o[4 * h + 2], o[4 * h + 3]);
            if constexpr (KIND == EPI_S8_HALF) flush_tile_s8_half(p.tile, C, ep.ldc, m0, n, p.M);
            else flush_tile<2>(p.tile, C, ep.ldc, m0, n, p.M);
        }
    }
}
// Runs body(IntConst<KIND>) for the call's output kind: the loop over a tile's whole chunks is instantiated per kind.  The chunks
// that are not whole (all of them for EPI_GENERAL) are left to the caller, who has one loop of epilogue_chunk for them.
template <bool S8_HALF, class Body>
__device__ __forceinline__ void for_epilogue_kind(int kind, bool i8, const Body& body) {
    switch (kind) {
        case EPI_F32: body(IntConst<EPI_F32>()); break;
        case EPI_BF16: body(IntConst<EPI_BF16>()); break;
        case EPI_S8: body(IntConst<EPI_S8>()); break;
        case EPI_S32: if (i8) body(IntConst<EPI_S32>()); break;
        case EPI_SILU: if (!i8) body(IntConst<EPI_SILU>()); break;
        case EPI_S8_HALF: if constexpr (S8_HALF) body(IntConst<EPI_S8_HALF>()); break;
        default: break;
    }
}

__device__ __forceinline__ unsigned cluster_ctarank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// shared::cluster address of the same shared-memory offset in CTA `rank` of the cluster
__device__ __forceinline__ unsigned mapa_rank(unsigned addr, unsigned rank) {
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void mbar_arrive_remote(unsigned cluster_addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void tma_load_2d_pair(unsigned dst, const CUtensorMap* map, unsigned leader_bar, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(map), "r"(leader_bar), "r"(x), "r"(y)
        : "memory");
}
__device__ __forceinline__ void tma_load_2d_pair_keep(unsigned dst, const CUtensorMap* map, unsigned leader_bar, int x, int y,
                                                      unsigned long long policy) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
        " [%0], [%1, {%3, %4}], [%2], %5;"
        ::"r"(dst), "l"(map), "r"(leader_bar), "r"(x), "r"(y), "l"(policy)
        : "memory");
}
// arrives on the barrier at the same offset of every CTA of the cluster whose bit is set in `mask`
__device__ __forceinline__ void tc_commit_mask(unsigned bar, unsigned short mask) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(bar), "h"(mask)
                 : "memory");
}
__device__ __forceinline__ void tc_commit_pair(unsigned bar) { tc_commit_mask(bar, (unsigned short)3); }
template <bool I8>
__device__ __forceinline__ void tc_mma_pair(unsigned d_tmem, unsigned long long adesc, unsigned long long bdesc,
                                            unsigned idesc, unsigned accumulate) {
    if constexpr (I8) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
            : "memory");
    } else {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
            : "memory");
    }
}

__device__ __forceinline__ unsigned bf16x2_sub(unsigned a, unsigned b) {
    const __nv_bfloat162 r = __hsub2(*(const __nv_bfloat162*)&a, *(const __nv_bfloat162*)&b);
    return *(const unsigned*)&r;
}
// two offset-binary weights u = v + 128 (bytes selected by sel, zero-extended) -> bf16x2 of v, exactly: 0x4300 | low 7 bits
// is 128 + low; 128 is taken off where bit 7 of u is set and 256 where it is not
__device__ __forceinline__ unsigned u8x2_to_bf16x2(unsigned w, unsigned sel) {
    const unsigned p = __byte_perm(w, 0u, sel);
    unsigned a, c;
    asm("lop3.b32 %0, %1, %2, %3, 0xea;" : "=r"(a) : "r"(p), "r"(0x007f007fu), "r"(0x43004300u));   // (p & m) | k
    asm("lop3.b32 %0, %1, %2, %3, 0xae;" : "=r"(c) : "r"(p), "r"(0x00800080u), "r"(0x43004300u));   // (~p & m) | k
    return bf16x2_sub(a, c);
}
// The same divided by 64, exactly, in two instructions: a byte u alone in a bf16 is the subnormal number u * 2^-133 (from 128 on with exponent
// field 1, which continues it without a step), and one fused multiply-add makes (u - 128) / 64 of it.
__device__ __forceinline__ unsigned u8x2_to_bf16x2_64th(unsigned w, unsigned sel) {
    unsigned r;
    asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(__byte_perm(w, 0u, sel)), "r"(0x7f007f00u), "r"(0xc000c000u));    // * 2^127 - 2
    return r;
}
// the eight nibbles n of a word -> four bf16x2 of (n - 8) / 64, exactly: nibbles at bits [4,8) and [20,24) need no shift, as the subnormal
// numbers 16 n * 2^-133
__device__ __forceinline__ void nib8_to_bf16x2_64th(unsigned w, unsigned* r) {
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const unsigned v = w >> (8 * h);
        asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(r[2 * h]) : "r"(v & 0x000f000fu), "r"(0x7f007f00u), "r"(0xbe00be00u));          // * 2^127 - 1/8
        asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(r[2 * h + 1]) : "r"(v & 0x00f000f0u), "r"(0x7d007d00u), "r"(0xbe00be00u));      // * 2^123 - 1/8
    }
}
// Arrival of a widening warp of the second CTA on the leader's barrier.  The bytes are handed over by the warp's proxy fence, which orders
// them before what the async proxy reads from then on, and the MMA that reads them is issued behind the leader's wait, which
// acquires at cluster scope.  The arrival itself has the default (CTA) scope: the form that CUTLASS has for the same hand-over
// of transformed operands to a two-CTA MMA (ClusterBarrier::arrive(cta_id) behind fence_view_async_shared).  A release at cluster
// scope is a full memory barrier at every slab: in each widening warp 36.7 us for 4 bits, 100 x 4096 x 11008 (26.6 without); in one
// forwarding warp of the second CTA 38.1 us for int8, 705 x 2560 x 10240 (32.1) and 157 us for 300 x 11008 x 8192 (100).
__device__ __forceinline__ void mbar_arrive_leader(unsigned cluster_addr) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void st_cluster_v4(unsigned cluster_addr, unsigned a, unsigned b, unsigned c, unsigned d) {
    asm volatile("st.shared::cluster.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(cluster_addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
// nibbles n at bits [0,4) and [16,20) of w -> bf16x2 of n - 8, exactly: (128 + n) - 136
__device__ __forceinline__ unsigned nib2_to_bf16x2(unsigned w) {
    unsigned a;
    asm("lop3.b32 %0, %1, %2, %3, 0xea;" : "=r"(a) : "r"(w), "r"(0x000f000fu), "r"(0x43004300u));
    return bf16x2_sub(a, 0x43084308u);
}

// ---- host side -----------------------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* sym = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)sym;
    }
    return fn;
}

// 2-D K-major tensor map: inner dimension = K elements, outer = rows; box = {128 bytes of K, box_rows}.
int make_map(CUtensorMap* map, const void* base, bool i8, uint64_t k_elems, uint64_t rows, uint64_t ld_bytes,
             uint32_t box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) { set_error("cuTensorMapEncodeTiled entry point not available"); return B200FC_ERR_CUDA; }
    cuuint64_t dims[2] = {k_elems, rows};
    cuuint64_t strides[1] = {ld_bytes};
    cuuint32_t box[2] = {(cuuint32_t)(i8 ? SLAB_BYTES : SLAB_BYTES / 2), box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(map, i8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (void*)base, dims,
                    strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { set_error("cuTensorMapEncodeTiled failed (%d)", (int)r); return B200FC_ERR_CUDA; }
    return B200FC_OK;
}

// How the epilogue may store whole chunks of the output: 1 = 16-byte pieces; 2 = int8 rows of an 8-bit GEMM in 8-byte pieces (widths that are a
// multiple of 8 only; single bytes took 28.7 us for int8 1559 x 1408 x 1240, 11.9 in pieces); 0 = element by element.
int output_vec(const Epilogue& ep, int n0, bool i8) {
    const int es = ep.out_dtype == B200FC_F32 || ep.out_dtype == B200FC_S32 ? 4 : (ep.out_dtype == B200FC_BF16 ? 2 : 1);
    const uintptr_t rows = (uintptr_t)ep.C | (uintptr_t)ep.ldc;
    if (ep.steps & B200FC_STEP_SILU_MUL) return (rows & 15) == 0 && n0 % 32 == 0;
    if (((rows | (uintptr_t)(n0 * es)) & 15) == 0) return 1;
    return i8 && ep.out_dtype == B200FC_S8 && ((rows | (uintptr_t)n0) & 7) == 0 ? 2 : 0;
}

// tcgen05 instruction descriptor (dense, K-major A and B, M = 128): accumulator format bits [4,6), A format [7,10),
// B format [10,13), N >> 3 at [17,23), M >> 4 at [24,29).
unsigned make_idesc(bool i8, bool a_signed, bool b_signed, int bn, int mma_m = BM) {
    unsigned d = 0;
    if (i8) {
        d |= 2u << 4;                       // int32 accumulator
        d |= (a_signed ? 1u : 0u) << 7;     // 8-bit integer: 1 = signed, 0 = unsigned
        d |= (b_signed ? 1u : 0u) << 10;
    } else {
        d |= 1u << 4;                       // fp32 accumulator
        d |= 1u << 7;                       // bf16
        d |= 1u << 10;
    }
    d |= (unsigned)(bn >> 3) << 17;
    d |= (unsigned)(mma_m >> 4) << 24;
    return d;
}

int num_sms() {
    static std::atomic<int> cache[64];   // SM count per device ordinal (0 = not asked yet)
    int dev = 0;
    cudaGetDevice(&dev);
    int n = cache[dev & 63].load(std::memory_order_relaxed);
    if (!n) {
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        if (n <= 0) n = 148;
        cache[dev & 63].store(n, std::memory_order_relaxed);
    }
    // the persistent GEMM grids take one CTA per SM; a caller that overlaps a collective with them leaves it a few SMs
    const int lim = sm_limit();
    return (lim >= 2 && lim < n) ? (lim & ~1) : n;
}

}  // namespace

}  // namespace b200fc
