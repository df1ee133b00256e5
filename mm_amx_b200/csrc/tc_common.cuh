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

// staging tiles of the four epilogue warps: 32 rows x 32 four-byte columns each, rows padded to 33 words
constexpr int EPI_TILE_WORDS = 32 * 33;

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
__device__ __forceinline__ bool mbar_try_wait(unsigned bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait.  Returns false when the CTA is aborting (this wait or another role's ran out of time).
// The clock is read after a batch of failed attempts only: a read of %globaltimer takes most of a microsecond, and one in front of
// the second attempt put that on every slab of a main loop whose loads are not always early (0.46 us per slab whatever its size).
// SLEEP_NS > 0: back off between polls (for waits that are long and not latency critical: the epilogue warps wait most
// of a tile's main loop, and five spinning warps cost issue slots and power that the tensor pipe could use).
template <int SLEEP_NS = 0>
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity, volatile int* abort_flag, unsigned long long limit) {
    if (mbar_try_wait(bar, parity)) return true;
    unsigned long long t0 = 0;
    while (true) {
#pragma unroll 1
        for (int i = 0; i < 16; i++) {
            if (SLEEP_NS > 0) __nanosleep(SLEEP_NS);
            if (mbar_try_wait(bar, parity)) return true;
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
// One lane of a converged warp, the same one every time.  The issuing loops below run as whole warps and elect the lane only
// around the TMA / MMA / commit instructions: these take their operands from uniform registers, which the compiler can keep
// them in only while the control flow is warp-uniform.  With the loop inside `if (lane == 0)` every MMA cost about 100 clocks of
// issue and every slab 480 more (880 clocks per 128 bytes of K however few columns a tile has).
__device__ __forceinline__ bool elect_one() {
    unsigned ok;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok));
    return ok != 0;
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
    const Epilogue* ep;
    int vec_ok, acc_is_int, n1;
    int M;             // rows of the output
    unsigned* tile;    // this warp's staging tile in shared memory (EPI_TILE_WORDS words)
    // the chunk's 32 per-column values, staged in shared memory ahead of the tile (16-byte aligned), or null: read
    // them from global memory
    const float* cv_deq = nullptr;
    const float* cv_bias = nullptr;
    const float* cv_q = nullptr;
};
// 32 rows x 32 four-byte values, one row per lane in registers -> global memory with full-line stores: the tile goes
// through shared memory and comes back with eight lanes per row (16 bytes each), so that one store instruction writes
// four whole 128-byte row segments instead of 32 scattered 16-byte pieces.  Both passes use 16-byte accesses: row r
// keeps its 16-byte piece j at position j ^ (r & 7), which makes the eight lanes of every shared-memory wavefront hit
// eight different bank groups on the way in (lanes = rows) and on the way out (lanes = pieces of one row).
// Called by all lanes of the warp; `tile` is 16-byte aligned.
__device__ __forceinline__ void store_tile_4b(const unsigned (&val)[32], unsigned* tile, char* C, long long ldc, int m, int n,
                                              int M) {
    const int lane = threadIdx.x & 31, m0 = m - lane;
    uint4* t4 = (uint4*)tile;
#pragma unroll
    for (int j = 0; j < 8; j++)
        t4[lane * 8 + (j ^ (lane & 7))] = make_uint4(val[4 * j], val[4 * j + 1], val[4 * j + 2], val[4 * j + 3]);
    __syncwarp();
    const int piece = lane & 7;
#pragma unroll
    for (int it = 0; it < 8; it++) {
        const int rr = it * 4 + (lane >> 3);
        const uint4 q = t4[rr * 8 + (piece ^ (rr & 7))];
        if (m0 + rr < M) *(uint4*)(C + (long long)(m0 + rr) * ldc + (long long)(n + piece * 4) * 4) = q;
    }
    __syncwarp();
}
// The same for rows of 64 bytes (32 bf16; val[j] = 4-byte words of the lane's row) and of 32 bytes (32 int8, or 16 bf16):
// one store instruction writes 8 / 16 whole row segments, where direct stores wrote 32 half sectors.  `c0` = the row
// segment's byte offset inside an output row.  Piece j of row r sits at j ^ ((r >> 1) & 3) / j ^ ((r >> 2) & 1): no conflicts.
__device__ __forceinline__ void store_tile_64(const unsigned (&val)[16], unsigned* tile, char* C, long long ldc, int m, long long c0, int M) {
    const int lane = threadIdx.x & 31, m0 = m - lane;
    uint4* t4 = (uint4*)tile;
#pragma unroll
    for (int j = 0; j < 4; j++)
        t4[lane * 4 + (j ^ ((lane >> 1) & 3))] = make_uint4(val[4 * j], val[4 * j + 1], val[4 * j + 2], val[4 * j + 3]);
    __syncwarp();
    const int piece = lane & 3;
#pragma unroll
    for (int it = 0; it < 4; it++) {
        const int rr = it * 8 + (lane >> 2);
        const uint4 q = t4[rr * 4 + (piece ^ ((rr >> 1) & 3))];
        if (m0 + rr < M) *(uint4*)(C + (long long)(m0 + rr) * ldc + c0 + piece * 16) = q;
    }
    __syncwarp();
}
__device__ __forceinline__ void store_tile_32(const unsigned (&val)[8], unsigned* tile, char* C, long long ldc, int m, long long c0, int M) {
    const int lane = threadIdx.x & 31, m0 = m - lane;
    uint4* t4 = (uint4*)tile;
#pragma unroll
    for (int j = 0; j < 2; j++)
        t4[lane * 2 + (j ^ ((lane >> 2) & 1))] = make_uint4(val[4 * j], val[4 * j + 1], val[4 * j + 2], val[4 * j + 3]);
    __syncwarp();
    const int piece = lane & 1;
#pragma unroll
    for (int it = 0; it < 2; it++) {
        const int rr = it * 16 + (lane >> 1);
        const uint4 q = t4[rr * 2 + (piece ^ ((rr >> 2) & 1))];
        if (m0 + rr < M) *(uint4*)(C + (long long)(m0 + rr) * ldc + c0 + piece * 16) = q;
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
// gelu_erf_poly (common.cuh) on two values: the same operations in the same order, the polynomial two values at a time
__device__ __forceinline__ f32x2 gelu_erf_poly2(f32x2 v) {
    constexpr unsigned coef[15] = {0x1f1c83fdu, 0xa3198977u, 0x268a7927u, 0xa998c963u, 0x2c67ddb2u, 0xaf013b2cu, 0x315d4a4fu,
                                   0xb3969b11u, 0x35a776e9u, 0xb79b0914u, 0x3970b255u, 0xbb1b7399u, 0x3ca3621fu, 0xbe082bc7u,
                                   0x3f4c4228u};
    const f32x2 x2 = mul2(v, v), xh = mul2(v, pack2(0.5f, 0.5f));
    f32x2 q = pack2(__uint_as_float(coef[0]), __uint_as_float(coef[0]));
#pragma unroll
    for (int i = 1; i < 15; i++) q = fma2(q, x2, pack2(__uint_as_float(coef[i]), __uint_as_float(coef[i])));
    q = mul2(fma2(q, v, pack2(1.0f, 1.0f)), xh);
    float x[2], h[2], y[2];
    unpack2(v, x[0], x[1]);
    unpack2(xh, h[0], h[1]);
    unpack2(q, y[0], y[1]);
#pragma unroll
    for (int e = 0; e < 2; e++) {
        float far;      // x < -5 -> 0, x > 5 -> x, NaN -> NaN
        asm("max.NaN.f32 %0, %1, 0f00000000;" : "=f"(far) : "f"(x[e]));
        const float ax = fabsf(x[e]);
        if (!(ax <= 5.0f)) y[e] = far;
        if (ax <= __uint_as_float(0x33800000u)) y[e] = h[e];
    }
    return pack2(y[0], y[1]);
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
// the 32 per-column values vec[n .. n + 32) of a chunk (every lane needs all of them): eight 16-byte loads when the
// chunk is whole and the vector 16-byte aligned, else 32 scalar loads clamped to the last valid column
__device__ __forceinline__ void load_col_vec(const float* __restrict__ vec, int n, int n1, float (&out)[32]) {
    if (n + 32 <= n1 && (((uintptr_t)(vec + n)) & 15) == 0) {
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const float4 t = __ldg((const float4*)(vec + n) + j);
            out[4 * j] = t.x; out[4 * j + 1] = t.y; out[4 * j + 2] = t.z; out[4 * j + 3] = t.w;
        }
    } else {
#pragma unroll
        for (int j = 0; j < 32; j++) out[j] = __ldg(vec + min(n + j, n1 - 1));
    }
}
// the same 32 values from the warp's staged copy (every lane reads the same addresses: broadcasts)
__device__ __forceinline__ void load_col_vec(const float* staged, const float* __restrict__ vec, int n, int n1, float (&out)[32]) {
    if (staged) {
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const float4 t = ((const float4*)staged)[j];
            out[4 * j] = t.x; out[4 * j + 1] = t.y; out[4 * j + 2] = t.z; out[4 * j + 3] = t.w;
        }
    } else {
        load_col_vec(vec, n, n1, out);
    }
}
__device__ __forceinline__ void epilogue_chunk(const unsigned (&r)[32], int m, int n, const EpiArgs p, bool row_ok,
                                               long long c_offset = 0) {
    const Epilogue& ep = *p.ep;
    const bool staged = p.vec_ok && n + 32 <= p.n1 && !ep.mc_reduce;   // warp-uniform
    char* Cb = (char*)ep.C + c_offset;
    if (ep.out_dtype == B200FC_S32 && staged) {
        store_tile_4b(r, p.tile, Cb, ep.ldc, m, n, p.M);
        return;
    }
    if (!row_ok && !staged) return;   // (rows beyond M take part in the staged stores' shuffle through shared memory)
    char* crow = (char*)ep.C + c_offset + (long long)m * ep.ldc;
    if (ep.out_dtype == B200FC_S32) {  // raw accumulators
        for (int j = 0; j < 32; j++)
            if (n + j < p.n1) ((int*)crow)[n + j] = (int)r[j];
        return;
    }
    float v[32];
#pragma unroll
    for (int j = 0; j < 32; j++) v[j] = p.acc_is_int ? (float)(int)r[j] : __uint_as_float(r[j]);

    if (ep.mc_reduce) {
        // Fused all-reduce: C is a multicast mapping of the output on every GPU of the tensor-parallel group; the
        // NVSwitch adds this rank's contribution into all replicas (multimem.red), so no separate collective runs.
        const bool full = p.vec_ok && n + 32 <= p.n1;
        if (ep.out_dtype == B200FC_F32) {
            float* dst = (float*)(crow + (long long)n * 4);
            if (full) {
#pragma unroll
                for (int j = 0; j < 8; j++)
                    asm volatile("multimem.red.relaxed.sys.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst + 4 * j),
                                 "f"(v[4 * j]), "f"(v[4 * j + 1]), "f"(v[4 * j + 2]), "f"(v[4 * j + 3])
                                 : "memory");
            } else {
                for (int j = 0; j < 32; j++)
                    if (n + j < p.n1) asm volatile("multimem.red.relaxed.sys.global.add.f32 [%0], %1;" ::"l"(dst + j), "f"(v[j]) : "memory");
            }
        } else {
            unsigned short* dst = (unsigned short*)(crow + (long long)n * 2);
            if (full) {
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    unsigned o[4];
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        __nv_bfloat162 h = __floats2bfloat162_rn(v[8 * j + 2 * q], v[8 * j + 2 * q + 1]);
                        o[q] = *(unsigned*)&h;
                    }
                    asm volatile("multimem.red.relaxed.sys.global.add.v4.bf16x2 [%0], {%1, %2, %3, %4};" ::"l"(dst + 8 * j),
                                 "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3])
                                 : "memory");
                }
            } else {
                for (int j = 0; j < 32; j += 2)   // the launcher guarantees an even column range for this mode
                    if (n + j + 1 < p.n1) {
                        __nv_bfloat162 h = __floats2bfloat162_rn(v[j], v[j + 1]);
                        asm volatile("multimem.red.relaxed.sys.global.add.bf16x2 [%0], %1;" ::"l"(dst + j), "r"(*(unsigned*)&h) : "memory");
                    }
            }
        }
        return;
    }

    if (ep.steps & B200FC_STEP_SILU_MUL) {
        // columns [0,16) gate, [16,32) up of the same 16 channels -> 16 bf16 outputs at column n/2
        float y[16];
#pragma unroll
        for (int j = 0; j < 16; j++) y[j] = silu_f(v[j]) * v[16 + j];
        if (staged) {
            unsigned o[8];
#pragma unroll
            for (int j = 0; j < 8; j++) {
                __nv_bfloat162 h = __floats2bfloat162_rn(y[2 * j], y[2 * j + 1]);
                o[j] = *(unsigned*)&h;
            }
            store_tile_32(o, p.tile, Cb, ep.ldc, m, n, p.M);      // column n / 2, two bytes each
        } else {
            unsigned short* dst = (unsigned short*)crow + (n >> 1);
            for (int j = 0; j < 16; j++)
                if (n + 16 + j < p.n1) dst[j] = f32_to_bf16_bits(y[j]);
        }
        return;
    }

    {
        f32x2 w[16];
#pragma unroll
        for (int j = 0; j < 16; j++) w[j] = pack2(v[2 * j], v[2 * j + 1]);
        // v = v * cv[j] (or * one scale), v + cv[j]
        auto scale_by = [&](const float* staged_cv, const float* vec, float one) {
            if (vec) {
                float sc[32];
                load_col_vec(staged_cv, vec, n, p.n1, sc);
#pragma unroll
                for (int j = 0; j < 16; j++) w[j] = mul2(w[j], mul2(pack2(one, one), pack2(sc[2 * j], sc[2 * j + 1])));
            } else {
#pragma unroll
                for (int j = 0; j < 16; j++) w[j] = mul2(w[j], pack2(one, one));
            }
        };
        if (ep.steps & B200FC_STEP_DEQUANT) scale_by(p.cv_deq, ep.deq_per_oc, ep.deq_scale);
        if (ep.steps & B200FC_STEP_BIAS) {
            float bs[32];
            load_col_vec(p.cv_bias, ep.bias, n, p.n1, bs);
#pragma unroll
            for (int j = 0; j < 16; j++) w[j] = add2(w[j], pack2(bs[2 * j], bs[2 * j + 1]));
        }
        if (ep.steps & B200FC_STEP_GELU) {
#pragma unroll
            for (int j = 0; j < 16; j++) w[j] = gelu_erf_poly2(w[j]);
        }
        if (ep.steps & B200FC_STEP_QUANT) scale_by(p.cv_q, ep.q_per_oc, ep.q_per_oc ? 1.0f : ep.q_scale);
#pragma unroll
        for (int j = 0; j < 16; j++) unpack2(w[j], v[2 * j], v[2 * j + 1]);
    }
    const bool full = p.vec_ok && n + 32 <= p.n1;
    if (ep.residual && row_ok) {
        // residual added in fp32, before the one rounding of the output
        const char* rrow = (const char*)ep.residual + (long long)m * ep.ld_res;
        if (full && (((uintptr_t)rrow + (size_t)n * 2) & 15) == 0) {
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int4 t = __ldg((const int4*)(rrow + (long long)n * 2) + q);
                const unsigned w4[4] = {(unsigned)t.x, (unsigned)t.y, (unsigned)t.z, (unsigned)t.w};
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    v[8 * q + 2 * e] += __uint_as_float(w4[e] << 16);
                    v[8 * q + 2 * e + 1] += __uint_as_float(w4[e] & 0xffff0000u);
                }
            }
        } else {
#pragma unroll
            for (int j = 0; j < 32; j++)
                v[j] += __uint_as_float((unsigned)((const unsigned short*)rrow)[min(n + j, p.n1 - 1)] << 16);
        }
    }
    if (ep.out_dtype == B200FC_F32) {
        if (staged) {
            unsigned u[32];
#pragma unroll
            for (int j = 0; j < 32; j++) u[j] = __float_as_uint(v[j]);
            store_tile_4b(u, p.tile, Cb, ep.ldc, m, n, p.M);
        } else {
            for (int j = 0; j < 32; j++)
                if (n + j < p.n1) ((float*)crow)[n + j] = v[j];
        }
    } else if (ep.out_dtype == B200FC_BF16) {
        if (staged) {
            unsigned o[16];
#pragma unroll
            for (int j = 0; j < 16; j++) {
                __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
                o[j] = *(unsigned*)&h;
            }
            store_tile_64(o, p.tile, Cb, ep.ldc, m, (long long)n * 2, p.M);
        } else {
            for (int j = 0; j < 32; j++)
                if (n + j < p.n1) ((unsigned short*)crow)[n + j] = f32_to_bf16_bits(v[j]);
        }
    } else {  // int8
        if (staged) {
            unsigned o[8];
#pragma unroll
            for (int j = 0; j < 8; j++) o[j] = f32x4_to_s8x4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
            store_tile_32(o, p.tile, Cb, ep.ldc, m, n, p.M);
        } else {
            for (int j = 0; j < 32; j++)
                if (n + j < p.n1) ((signed char*)crow)[n + j] = (signed char)f32_to_s8(v[j]);
        }
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
