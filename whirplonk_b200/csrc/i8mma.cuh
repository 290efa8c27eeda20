// i8mma.cuh -- exact 8-bit contractions on the tensor cores (tcgen05.mma
// kind::i8, u8 x u8 -> s32): operands, tensor memory, byte constants, and the
// reduction of byte sums mod p.  Used by the encoder's DFT passes (k_dft8.cu)
// and the STIR covector update (k_cov_gemm.cu).
#pragma once
#include "gl.cuh"

namespace wg {

// One operand block: 128 rows of 128 bytes (16 words).
constexpr u32 BLK = 128 * 128;

__device__ __forceinline__ u32 smem_u32(const void* p) { return (u32)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void mbar_init(u32 bar, u32 count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(u32 bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Waits for the phase; gives up after about two seconds (a contraction takes
// microseconds) and reports it.
__device__ __forceinline__ bool mbar_wait(u32 bar, u32 parity) {
    u32 done = 0;
    unsigned long long t0 = 0;
    for (u32 it = 0; it < (1u << 28); ++it) {
        asm volatile("{\n\t.reg .pred p;\n\t"
                     "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(done)
                     : "r"(bar), "r"(parity)
                     : "memory");
        if (done) return true;
        if ((it & 63) == 63) {
            unsigned long long t;
            asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
            if (!t0) t0 = t;
            else if (t - t0 > 2000000000ull) return false;
        }
    }
    return false;
}
// The producer of a ring of bulk copies, before it leaves: the copies of the last
// `armed` stages filled (the next one would be stage s in phase ph) have landed, so
// the CTA's shared memory outlives them even when the consumers gave up.  Behind
// consumers that did not, it waits for nothing.
__device__ __forceinline__ bool ring_drain(u32 full, u32 stages, u32 s, u32 ph, u32 armed) {
    bool ok = true;
    for (; armed > 0; --armed) {
        if (s == 0) s = stages, ph ^= 1;
        --s;
        ok = mbar_wait(full + 8 * s, ph) && ok;
    }
    return ok;
}

// K-major shared-memory operand, rows of 128 bytes in 8-row atoms of 1024
// bytes, 128-byte swizzle (16-byte chunk c of row r at chunk c ^ (r mod 8)).
__device__ __forceinline__ u64 op_desc(u32 addr) {
    return (u64)((addr & 0x3FFFFu) >> 4) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
// D s32, A and B unsigned bytes, both K-major, M = 128.
__device__ __forceinline__ constexpr u32 op_idesc(u32 n) { return (2u << 4) | ((n >> 3) << 17) | (8u << 24); }
__device__ __forceinline__ void mma_i8(u32 d, u64 a, u64 b, u32 idesc, u32 acc) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
                 "l"(a), "l"(b), "r"(idesc), "r"(acc)
                 : "memory");
}
// 128 rows x 128 bytes times n byte sums: four instructions of 32 bytes of K.
__device__ __forceinline__ void mma_block(u32 d, u32 a, u32 b, u32 n) {
    const u64 da = op_desc(a), db = op_desc(b);
#pragma unroll
    for (u32 k = 0; k < 4; ++k) mma_i8(d, da + 2 * k, db + 2 * k, op_idesc(n), k);
}
__device__ __forceinline__ void mma_commit(u32 bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// The byte sums of NB consecutive outputs (this thread's row): 8 NB registers.
template <int NB>
struct Limbs {
    u32 l[8 * NB];
};
#define WG_R8(x, o) "=r"(x[o]), "=r"(x[o + 1]), "=r"(x[o + 2]), "=r"(x[o + 3]), "=r"(x[o + 4]), "=r"(x[o + 5]), "=r"(x[o + 6]), "=r"(x[o + 7])
#define WG_P8(x, o) "+r"(x[o]), "+r"(x[o + 1]), "+r"(x[o + 2]), "+r"(x[o + 3]), "+r"(x[o + 4]), "+r"(x[o + 5]), "+r"(x[o + 6]), "+r"(x[o + 7])
__device__ __forceinline__ void tm_ld(u32 addr, Limbs<1>& x) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];" : WG_R8(x.l, 0) : "r"(addr));
}
__device__ __forceinline__ void tm_ld(u32 addr, Limbs<2>& x) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : WG_R8(x.l, 0), WG_R8(x.l, 8)
                 : "r"(addr));
}
__device__ __forceinline__ void tm_ld(u32 addr, Limbs<4>& x) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                 "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                 : WG_R8(x.l, 0), WG_R8(x.l, 8), WG_R8(x.l, 16), WG_R8(x.l, 24)
                 : "r"(addr));
}
// Waits for this thread's tensor-memory loads.
__device__ __forceinline__ void tm_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// The loaded registers pass through here after the wait, so nothing that reads
// them is scheduled before it.
template <int NB>
__device__ __forceinline__ void tm_pin(Limbs<NB>& x) {
#pragma unroll
    for (int k = 0; k < NB; ++k) asm volatile("" : WG_P8(x.l, 8 * k));
}

// Two digits of base 2^32, each below 2^52: value = w0 + 2^32 w1.
struct W2 {
    u64 w0, w1;
};
__device__ __forceinline__ u64 madw(u32 a, u32 b, u64 c) {
    u64 d;
    asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
    return d;
}
// w0 + 2^32 w1 (digits below 2^60) as some 64-bit representative mod p (2^64 = 2^32 - 1).
__device__ __forceinline__ u64 w_reduce(const W2& x) {
    u64 s;
    asm("{\n\t.reg .u32 l0, l1, t0, t1, m0, m1, c;\n\t.reg .u64 h, m;\n\t"
        "mov.b64 {l0, l1}, %1;\n\t"
        "mov.b64 {t0, t1}, %2;\n\t"
        "add.cc.u32 t0, t0, l1;\n\t"
        "addc.u32 t1, t1, 0;\n\t"  // value = l0 + 2^32 t0 + 2^64 t1, t1 < 2^28
        "mul.wide.u32 m, t1, 0xFFFFFFFF;\n\t"
        "mov.b64 {m0, m1}, m;\n\t"
        "add.cc.u32 l0, l0, m0;\n\t"
        "addc.cc.u32 t0, t0, m1;\n\t"
        "addc.u32 c, 0, 0;\n\t"
        "mov.b64 h, {l0, t0};\n\t"
        "mad.wide.u32 %0, c, 0xFFFFFFFF, h;\n\t}"  // a carry leaves h < 2^61: no second one
        : "=l"(s)
        : "l"(x.w0), "l"(x.w1));
    return s;
}
__device__ __forceinline__ u64 gl_canon(u64 s) {
    u64 t = s + GL_EPS;  // wraps iff s >= p
    return t < GL_EPS ? t : s;
}
// The constant v as operand rows: row j (128 bytes each, from `rows`, a multiple
// of 1024 bytes) holds at word i the bytes byte_j(v 2^(8b) mod p), b = 0 .. 7 --
// eight representatives of v 2^(8b), transposed.
__device__ __forceinline__ void expand_bytes(u64 v, unsigned char* rows, u32 i) {
    u32 w0[8], w1[8];
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        w0[b] = (u32)v;
        w1[b] = (u32)(v >> 32);
        const u64 s = v << 8, t = s + (v >> 56) * GL_EPS;  // 2^8 v
        v = t < s ? t + GL_EPS : t;
    }
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int g = 0; g < 4; ++g) {  // byte j = 4 h + g of the eight values
            u32 x[2];
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const u32* w = h ? w1 : w0;
                const u32 sel = g | (4 + g) << 4;
                const u32 p = __byte_perm(w[4 * c], w[4 * c + 1], sel), s = __byte_perm(w[4 * c + 2], w[4 * c + 3], sel);
                x[c] = __byte_perm(p, s, 0x5410);
            }
            const u32 j = 4 * h + g;
            *reinterpret_cast<u64*>(rows + j * 128 + (((i >> 1) ^ j) << 4) + (i & 1) * 8) = (u64)x[1] << 32 | x[0];
        }
}

}  // namespace wg
