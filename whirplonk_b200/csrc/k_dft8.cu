// k_dft8.cu -- the LDE's transform as exact 8-bit contractions on the tensor cores.
//
// A Goldilocks word is eight bytes, x = sum_b x_b 2^(8b), so a DFT over R words
// is an integer contraction over 8 R bytes:
//     X[a] = sum_(i,b) x_(i,b) v_(a,i,b),   v_(a,i,b) = w^(a i) 2^(8b) mod p,
// and with v split into its own bytes the tensor cores (tcgen05.mma kind::i8,
// u8 x u8 -> s32, exact) return for every output the eight sums
//     l_j = sum_(i,b) x_(i,b) byte_j(v_(a,i,b)) <= 128 * 255^2 < 2^23
// over one block of 16 words, with X[a] = sum_j l_j 2^(8j) (mod p).  The CUDA
// cores only join eight 23-bit sums into one word (~13 instructions), instead
// of the 4 x 46 instructions of four radix-2 stages.
//
// A word in memory already is its eight bytes in order, so the message itself
// is the contraction's A operand: a row is one transform (column, tile lane),
// its K bytes are 16 consecutive words of it.  B holds the bytes of the
// constants, built in shared memory by each CTA (k_dft8 `build_b`).
//
// A radix of 32 or 64 splits its words by residue mod 2 or 4 into blocks of
// 16: X[a + 16 s] = sum_r w_(2^e)^(r s) Y_r[a] with the block twiddles w^(a r)
// inside B, so the extra one or two levels are the additions of a radix-2 / 4
// butterfly on unreduced sums (w_4 = 2^48 is a shift).  That keeps 1024 byte
// products per output whatever the radix (a plain 64-point contraction has
// 4096, and its constants fill 256 KB).
//
// What bounds it: the integer pipes again (45-60 instructions per output and
// round: join 13-20, factor 17, addresses and shared memory), then HBM for the
// pass boundaries; the contraction itself takes 1/8 clock per output and SM (a
// sixth of the time).  Measured on B200 against the butterfly passes of
// k_ntt.cu, 16 planes 2^20 -> 2^22: 923 us against 1658; 48 planes 2^16 -> 2^21:
// 1157 against 1846; 48 planes 2^12 -> 2^20: 435 against 752.
#include <algorithm>

#include "gl.cuh"
#include "launch.h"
#include "transcript.cuh"

namespace wg {

namespace {

constexpr int TEAMS = 2;             // independent halves of a CTA: one's contraction runs under the other's joins
constexpr int TEAM_WARPS = 8;
constexpr int TT = 32 * TEAM_WARPS;  // threads of a team
constexpr int WGS = TEAM_WARPS / 4;  // warpgroups of a team: each reads all 128 rows, 1 / WGS of the outputs
constexpr u32 BLK = 128 * 128;       // bytes of one operand block: 128 rows x 16 words (A), 128 byte sums x 128 bytes (B)
constexpr u32 TEAM_COLS = 256;       // tensor-memory columns of a team

// 64-bit address-space helpers.
__device__ __forceinline__ u32 smem_u32(const void* p) { return (u32)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void cp8(u32 dst, const u64* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void team_sync(u32 team) { asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "n"(TT) : "memory"); }
// The barrier with an OR: every thread of the team gets the same answer.
__device__ __forceinline__ bool team_any(u32 team, bool v) {
    u32 r;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.or.pred q, %2, %3, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                 : "=r"(r)
                 : "r"((u32)v), "r"(team + 1), "n"(TT)
                 : "memory");
    return r != 0;
}

__device__ __forceinline__ void sts64(u32 a, u64 v) { asm volatile("st.shared.u64 [%0], %1;" ::"r"(a), "l"(v) : "memory"); }
__device__ __forceinline__ u64 lds64(u32 a) {
    u64 v;
    asm volatile("ld.shared.u64 %0, [%1];" : "=l"(v) : "r"(a) : "memory");
    return v;
}

__device__ __forceinline__ void mbar_init(u32 bar) { asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory"); }
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

// The eight byte sums of one output (this thread's row).
struct Limbs {
    u32 l[8];
};
__device__ __forceinline__ void tm_ld(u32 addr, Limbs& x) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(x.l[0]), "=r"(x.l[1]), "=r"(x.l[2]), "=r"(x.l[3]), "=r"(x.l[4]), "=r"(x.l[5]), "=r"(x.l[6]),
                   "=r"(x.l[7])
                 : "r"(addr));
}
// The loaded registers pass through the wait, so nothing that reads them is
// scheduled before it.
__device__ __forceinline__ void tm_wait(Limbs& x) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(x.l[0]), "+r"(x.l[1]), "+r"(x.l[2]), "+r"(x.l[3]), "+r"(x.l[4]), "+r"(x.l[5]), "+r"(x.l[6]),
                   "+r"(x.l[7]));
}
__device__ __forceinline__ void tm_pin(Limbs& x) {
    asm volatile("" : "+r"(x.l[0]), "+r"(x.l[1]), "+r"(x.l[2]), "+r"(x.l[3]), "+r"(x.l[4]), "+r"(x.l[5]),
                      "+r"(x.l[6]), "+r"(x.l[7]));
}

// ---- joining the byte sums -------------------------------------------------
// u_j = l_(2j) + 2^8 l_(2j+1) <= 257 * 8323200 < 2^31: four digits of base 2^16.
struct U4 {
    u32 u[4];
};
__device__ __forceinline__ U4 join(const Limbs& x) {
    U4 r;
#pragma unroll
    for (int j = 0; j < 4; ++j) r.u[j] = x.l[2 * j] + (x.l[2 * j + 1] << 8);
    return r;
}
__device__ __forceinline__ U4 u_add(const U4& a, const U4& b) {  // < 2^32
    return U4{{a.u[0] + b.u[0], a.u[1] + b.u[1], a.u[2] + b.u[2], a.u[3] + b.u[3]}};
}
// Digits near 2^31 (so a difference of two u_j plus one stays in 32 bits)
// whose sum over 2^(16 j) is a multiple of p.
constexpr u64 U_MAX = 257ull * 8323200;
constexpr u32 u_bias(int j) {
    constexpr u32 B = 0x7F900000u;  // U_MAX <= B, B + 65535 + U_MAX < 2^32
    // (-B (1 + 2^16 + 2^32 + 2^48)) mod p, in 16-bit digits
    const unsigned __int128 s = (unsigned __int128)B * ((1ull << 48) + (1ull << 32) + (1ull << 16) + 1);
    const u64 r = GL_P - (u64)(s % GL_P);
    return B + (u32)((r >> (16 * j)) & 0xFFFF);
}
constexpr u32 UB0 = u_bias(0), UB1 = u_bias(1), UB2 = u_bias(2), UB3 = u_bias(3);
static_assert(UB0 >= U_MAX && UB1 >= U_MAX && UB2 >= U_MAX && UB3 >= U_MAX, "difference below zero");
static_assert(UB0 + U_MAX < (1ull << 32) && UB1 + U_MAX < (1ull << 32) && UB2 + U_MAX < (1ull << 32) &&
                  UB3 + U_MAX < (1ull << 32), "difference above 32 bits");
__device__ __forceinline__ U4 u_sub(const U4& a, const U4& b) {
    return U4{{a.u[0] - b.u[0] + UB0, a.u[1] - b.u[1] + UB1, a.u[2] - b.u[2] + UB2, a.u[3] - b.u[3] + UB3}};
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
__device__ __forceinline__ W2 u_w(const U4& a) { return W2{madw(a.u[1], 65536u, a.u[0]), madw(a.u[3], 65536u, a.u[2])}; }

// w0 + 2^32 w1 as some 64-bit representative mod p (2^64 = 2^32 - 1).
__device__ __forceinline__ u64 w_reduce(const W2& x) {
    u64 s;
    asm("{\n\t.reg .u32 l0, l1, t0, t1, m0, m1, c;\n\t.reg .u64 h, m;\n\t"
        "mov.b64 {l0, l1}, %1;\n\t"
        "mov.b64 {t0, t1}, %2;\n\t"
        "add.cc.u32 t0, t0, l1;\n\t"
        "addc.u32 t1, t1, 0;\n\t"  // value = l0 + 2^32 t0 + 2^64 t1, t1 < 2^21
        "mul.wide.u32 m, t1, 0xFFFFFFFF;\n\t"
        "mov.b64 {m0, m1}, m;\n\t"
        "add.cc.u32 l0, l0, m0;\n\t"
        "addc.cc.u32 t0, t0, m1;\n\t"
        "addc.u32 c, 0, 0;\n\t"
        "mov.b64 h, {l0, t0};\n\t"
        "mad.wide.u32 %0, c, 0xFFFFFFFF, h;\n\t}"  // a carry leaves h < 2^53: no second one
        : "=l"(s)
        : "l"(x.w0), "l"(x.w1));
    return s;
}
__device__ __forceinline__ u64 gl_canon(u64 s) {
    u64 t = s + GL_EPS;  // wraps iff s >= p
    return t < GL_EPS ? t : s;
}
// a b mod p for any 64-bit a, b: some 64-bit representative.
__device__ __forceinline__ u64 mul_nc(u64 a, u64 b) {
    u64 lo, hi, s;
    asm("mul.lo.u64 %0, %2, %3;\n\tmul.hi.u64 %1, %2, %3;" : "=l"(lo), "=l"(hi) : "l"(a), "l"(b));
    asm("{\n\t.reg .u32 l0, l1, h0, h1, t0, t1, m, c;\n\t.reg .u64 t, u;\n\t"
        "mov.b64 {l0, l1}, %1;\n\t"
        "mov.b64 {h0, h1}, %2;\n\t"
        "sub.cc.u32 t0, l0, h1;\n\t"
        "subc.cc.u32 t1, l1, 0;\n\t"
        "subc.u32 m, 0, 0;\n\t"
        "sub.cc.u32 t0, t0, m;\n\t"
        "subc.u32 t1, t1, 0;\n\t"
        "mov.b64 t, {t0, t1};\n\t"
        "mul.wide.u32 u, h0, 0xFFFFFFFF;\n\t"
        "add.cc.u64 %0, t, u;\n\t"
        "addc.u32 c, 0, 0;\n\t"
        "mad.wide.u32 %0, c, 0xFFFFFFFF, %0;\n\t}"
        : "=l"(s)
        : "l"(lo), "l"(hi));
    return s;
}

// The outputs X[a + 16 s], s < 2^E, from the blocks' sums for output a.
template <int E>
__device__ __forceinline__ void combine(const Limbs (&y)[1 << E], u64 (&x)[1 << E]) {
    if constexpr (E == 0) {
        x[0] = w_reduce(u_w(join(y[0])));
    } else if constexpr (E == 1) {
        const U4 a = join(y[0]), b = join(y[1]);
        x[0] = w_reduce(u_w(u_add(a, b)));
        x[1] = w_reduce(u_w(u_sub(a, b)));
    } else {
        const U4 a = join(y[0]), b = join(y[1]), c = join(y[2]), d = join(y[3]);
        const W2 e0 = u_w(u_add(a, c)), e1 = u_w(u_add(b, d));
        const W2 o0 = u_w(u_sub(a, c));
        const U4 o = u_sub(b, d);
        // 2^18 p = C0 + 2^32 C1 with both digits above any subtrahend below
        constexpr u64 C0 = (1ull << 18) + (1ull << 50), C1 = (1ull << 50) - (1ull << 19);
        // 2^48 o = 2^32 p1 - p0:  2^64 = 2^32 - 1, 2^80 = 2^48 - 2^16, 2^96 = -1
        const u64 z = madw(o.u[2], 65536u, o.u[1]);
        const u64 p0 = z + o.u[3], p1 = madw(o.u[0], 65536u, z);
        x[0] = w_reduce(W2{e0.w0 + e1.w0, e0.w1 + e1.w1});
        x[1] = w_reduce(W2{o0.w0 + C0 - p0, o0.w1 + C1 + p1});
        x[2] = w_reduce(W2{e0.w0 + C0 - e1.w0, e0.w1 + C1 - e1.w1});
        x[3] = w_reduce(W2{o0.w0 + C0 + p0, o0.w1 + C1 - p1});
    }
}

// w_{2^logM}^e from the two-level table of powers of w_{2^TW_LOG}.
__device__ __forceinline__ u64 root_pow(u64 e, u32 logM, const u64* hi, const u64* lo) {
    const u64 x = (e & ((1ull << logM) - 1)) << (TW_LOG - logM);
    return gl_mul(__ldg(reinterpret_cast<const unsigned long long*>(hi) + (x >> TW_HALF)),
                  __ldg(reinterpret_cast<const unsigned long long*>(lo) + (x & ((1ull << TW_HALF) - 1))));
}

// Constants of a round of radix 2^(4 + E) whose outputs are the powers
// q + 2^lE a of w = w_{2^(4 + E + lE)}: block r, row (a, j), bytes (i, b) hold
// byte j of w^((2^E i + r)(q + 2^lE a)) 2^(8b).  One thread per (r, a, i): eight
// representatives, transposed to eight words of bytes.
template <int E>
__device__ __forceinline__ void build_b(u32 smB, u32 q, u32 lE, const u64* hi, const u64* lo) {
    for (u32 k = threadIdx.x; k < (256u << E); k += TEAMS * TT) {
        const u32 i = k & 15, a = (k >> 4) & 15, r = k >> 8;
        u64 v = root_pow((u64)((i << E) + r) * (q + ((u64)a << lE)), 4 + E + lE, hi, lo);
        u32 w0[8], w1[8];
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            w0[b] = (u32)v;
            w1[b] = (u32)(v >> 32);
            const u64 s = v << 8, t = s + (v >> 56) * GL_EPS;  // 2^8 v
            v = t < s ? t + GL_EPS : t;
        }
        const u32 row = smB + r * BLK + a * 1024 + (i & 1) * 8;
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
                sts64(row + j * 128 + (((i >> 1) ^ j) << 4), (u64)x[1] << 32 | x[0]);
            }
    }
}

// Shared-memory byte of word d of row `row` in an operand of radix 2^(4 + E):
// word d is word d >> E of block d mod 2^E; rows in groups of 128.
template <int E>
__device__ __forceinline__ u32 op_addr(u32 row, u32 d) {
    const u32 i = d >> E, r = d & ((1u << E) - 1);
    return (((row >> 7) << E) + r) * BLK + (row & 127) * 128 + (((i >> 1) ^ (row & 7)) << 4) + ((i & 1) << 3);
}

struct Dft8Args {
    const u64* src[3];  // first pass: message planes (block b of component c at src[c] + b M1 M2)
    const u64* in;      // last pass: scratch planes
    u64* out;           // scratch planes (first), codeword planes (last)
    u32 depth, logN, lE, l1, l2;
    u32 tiles_per_q;    // tiles per coset q (first pass) or in all (last pass)
    u32 total;          // tiles
    const u64* tw_hi;
    const u64* tw_lo;
    const u64* tab;     // first pass: w_N^(row col), row-major in rows of 2^l2
    u32* err;
};

// One pass.  With N = 2^lE M1 M2, message index i = c2 + M2 c1, codeword index
// k = k1 + 2^lE M1 k2 and k1 = q + 2^lE a (q the coset):
//   first pass: S[k1][c2] = w_N^(c2 k1) sum_c1 x[c2 + M2 c1] w_{2^lE M1}^(c1 k1)
//   last pass:  X[k1 + 2^lE M1 k2] = sum_c2 S[k1][c2] w_{M2}^(c2 k2)
// The zero padding is never touched: the coset's factor w^(c1 q) sits in the
// constants of the first round.
// E2 < 0: the pass is one round of radix 2^(4 + E1) over `rows` independent
// transforms per tile (columns of all planes, flattened).  Otherwise two
// rounds, 2^(4 + E1) then 2^(4 + E2), of W transforms per tile, the tile's
// words staying in shared memory between them.
template <int E1, int E2, bool FIRST>
struct Cfg {
    static constexpr bool TWO = E2 >= 0;
    static constexpr int E2P = TWO ? E2 : 0;
    static constexpr int LR1 = 4 + E1, LR2 = 4 + E2P;
    static constexpr int L = TWO ? LR1 + LR2 : LR1;
    static constexpr int LT = !TWO && E1 == 2 ? 13 : 12;  // words of a team's tile
    static constexpr int LW = LT - L;                     // transforms of a tile
    static constexpr int UNITS1 = 1 << (LT - 7 - LR1);    // 128-row groups of round 1
    static constexpr int UNITS2 = 1 << (LT - 7 - LR2);
    static constexpr int HALVES = !TWO && E1 == 2 ? 2 : 1;  // outputs of a round in two turns of tensor memory
    static constexpr u32 DATA = 8u << LT;
    static constexpr u32 B1 = BLK << E1, B2 = TWO ? BLK << E2P : 0, TWB = TWO ? 8u << L : 0;
    static constexpr u32 SMEM = TEAMS * DATA + B1 + B2 + TWB + 1024 + 64;
};

template <int E1, int E2, bool FIRST>
__global__ void __launch_bounds__(TEAMS* TT, 1) k_dft8(const __grid_constant__ Dft8Args a) {
    using C = Cfg<E1, E2, FIRST>;
    extern __shared__ unsigned char smem_raw[];
    __shared__ u32 s_tmem;
    __shared__ __align__(8) u64 s_bar[TEAMS];
    const u32 base = (smem_u32(smem_raw) + 1023) & ~1023u;
    const u32 team = threadIdx.x / TT, tid = threadIdx.x % TT, warp = tid >> 5, lane = tid & 31;
    const u32 smD = base + team * C::DATA;
    const u32 smB1 = base + TEAMS * C::DATA, smB2 = smB1 + C::B1, smT = smB2 + C::B2;
    const u32 bar = smem_u32(&s_bar[team]);

    if (threadIdx.x < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)),
                     "n"(TEAMS * TEAM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) mbar_init(bar);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    tc_before();
    __syncthreads();
    tc_after();
    const u32 tmem = s_tmem + team * TEAM_COLS;
    const u32 tlane = tmem + ((warp & 3) << 21);  // this warp's 32 rows
    const u32 wgi = warp >> 2;
    const u32 trow = ((warp & 3) << 5) | lane;
    u32 phase = 0;
    bool ok = true;

    const u64 M2 = 1ull << a.l2;
    const u32 lN1 = a.logN - a.l2;  // 2^lE M1
    constexpr u32 W = 1u << C::LW;

    // Start the copies of tile t of coset q.
    auto load = [&](u32 t) {
#pragma unroll
        for (int j = 0; j < (1 << C::LT) / TT; ++j) {
            const u32 x = tid + j * TT;
            if constexpr (C::TWO) {
                // Bits of x from the lowest: the contiguous index of memory, then
                // the operand word's parity, so that a warp's 32 words fall on
                // all banks twice (the swizzle spreads rows mod 8).
                u32 w, i2, r2, i1, r1;
                if constexpr (FIRST) {
                    constexpr int Z = E1 + C::E2P;  // low bits of i2 in the lane
                    w = x & (W - 1);
                    i2 = (x >> C::LW) & ((1u << Z) - 1);
                    i1 = (x >> (C::LW + Z)) & 1;
                    u32 y = x >> (C::LW + Z + 1);
                    i2 |= (y & ((1u << (4 - Z)) - 1)) << Z;
                    y >>= 4 - Z;
                    r2 = y & ((1u << C::E2P) - 1);
                    y >>= C::E2P;
                    i1 |= (y & 7) << 1;
                    r1 = y >> 3;
                } else {
                    u32 d2 = x & 15;
                    i1 = (x >> 4) & 1;
                    u32 y = x >> 5;
                    d2 |= (y & ((1u << C::E2P) - 1)) << 4;
                    y >>= C::E2P;
                    i1 |= (y & 7) << 1;
                    y >>= 3;
                    r1 = y & ((1u << E1) - 1);
                    w = y >> E1;
                    r2 = d2 & ((1u << C::E2P) - 1);
                    i2 = d2 >> C::E2P;
                }
                const u32 d1 = (i1 << E1) | r1, d2 = (i2 << C::E2P) | r2;
                // row of (d2, w): the 16 words i2 of one block row of round 2 in
                // 16 lanes, permuted by w so that neighbouring transforms differ mod 8
                const u32 row = (((r2 << C::LW) | w) << 4) | (i2 ^ ((w << (E1 + C::E2P)) & 7));
                const u64* p;
                if constexpr (FIRST) {
                    const u32 rho = t << C::LW, plane = rho >> a.l2;
                    const u32 comp = plane / a.depth, blk = plane % a.depth;
                    const u64* s = comp == 0 ? a.src[0] : comp == 1 ? a.src[1] : a.src[2];
                    p = s + ((u64)blk << (a.l1 + a.l2)) + (((u64)(d2 + (d1 << C::LR2))) << a.l2) + (rho & (u32)(M2 - 1)) + w;
                } else {
                    p = a.in + ((((u64)t << C::LW) + w) << a.l2) + d2 + (d1 << C::LR2);
                }
                cp8(smD + op_addr<E1>(row, d1), p);
            } else {
                u32 row, d;
                const u64* p;
                if constexpr (FIRST) {
                    row = x & 15;
                    u32 i = (x >> 4) & 1;
                    u32 y = x >> 5;
                    row |= (y & ((W >> 4) - 1)) << 4;
                    y >>= C::LW - 4;
                    i |= (y & 7) << 1;
                    d = (i << E1) | (y >> 3);
                    const u32 rho = (t << C::LW) + row, plane = rho >> a.l2;
                    const u32 comp = plane / a.depth, blk = plane % a.depth;
                    const u64* s = comp == 0 ? a.src[0] : comp == 1 ? a.src[1] : a.src[2];
                    p = s + ((u64)blk << (a.l1 + a.l2)) + ((u64)d << a.l2) + (rho & (u32)(M2 - 1));
                } else {
                    // 16 consecutive words of a row and of the row 2^(1 - E1 ...) away,
                    // whose chunks the swizzle puts on the other banks
                    constexpr int RB = E1 == 0 ? 0 : E1 == 1 ? 2 : 1;
                    d = x & 15;
                    const u32 rb = (x >> 4) & 1;
                    u32 y = x >> 5;
                    d |= (y & ((1u << E1) - 1)) << 4;
                    y >>= E1;
                    row = (y & ((1u << RB) - 1)) | rb << RB | (y >> RB) << (RB + 1);
                    p = a.in + ((((u64)t << C::LW) + row) << a.l2) + d;
                }
                cp8(smD + op_addr<E1>(row, d), p);
            }
        }
    };

    const u32 lo_t = (u32)((u64)a.total * blockIdx.x / gridDim.x), hi_t = (u32)((u64)a.total * (blockIdx.x + 1) / gridDim.x);
    for (u32 cur = lo_t; cur < hi_t;) {
        const u32 q = FIRST ? cur / a.tiles_per_q : 0;
        const u32 t0 = cur - q * a.tiles_per_q;
        const u32 cnt = min(hi_t - cur, a.tiles_per_q - t0);
        const u32 t1 = t0 + cnt;
        cur += cnt;
        __syncthreads();  // every contraction of the previous coset is done
        u32 t = t0 + team;
        if (t < t1) load(t);
        const u32 lEq = FIRST ? a.lE : 0;
        build_b<E1>(smB1, q, lEq, a.tw_hi, a.tw_lo);
        if constexpr (C::TWO) {
            build_b<E2>(smB2, 0, 0, a.tw_hi, a.tw_lo);
            // inter-round factors w_{2^(L + lE)}^(d2 (q + 2^lE a)) at [a][r2][i2]
            for (u32 k = threadIdx.x; k < (1u << C::L); k += TEAMS * TT) {
                const u32 i2 = k & 15, r2 = (k >> 4) & ((1u << C::E2P) - 1), aa = k >> C::LR2;
                const u32 d2 = (i2 << C::E2P) | r2;
                sts64(smT + 8 * k, root_pow((u64)d2 * (q + ((u64)aa << lEq)), C::L + lEq, a.tw_hi, a.tw_lo));
            }
        }
        fence_async();
        __syncthreads();
        for (; t < t1; t += TEAMS) {
            cp_wait_all();
            fence_async();
            tc_before();
            if (team_any(team, !ok)) break;
            if constexpr (C::TWO) {
                if (tid == 0) {
                    tc_after();
#pragma unroll
                    for (int u = 0; u < C::UNITS1; ++u)
#pragma unroll
                        for (int r = 0; r < (1 << E1); ++r)
                            mma_block(tmem + ((u << E1) + r) * 128, smD + ((u << E1) + r) * BLK, smB1 + r * BLK, 128);
                    mma_commit(bar);
                }
                ok = ok && mbar_wait(bar, phase);
                phase ^= 1;
                tc_after();
                // Round 1 outputs a = a' + 16 s of row (d2, w): times the factor, to word d2 of row (a, w).
#pragma unroll
                for (int u = 0; u < C::UNITS1; ++u) {
                    const u32 row = u * 128 + trow, hi = row >> 4, w = hi & (W - 1), r2 = hi >> C::LW;
                    const u32 i2 = (row & 15) ^ ((w << (E1 + C::E2P)) & 7);
                    const u32 tcol = tlane + (u << E1) * 128 + wgi * (16 / WGS) * 8;
                    Limbs y[1 << E1];
#pragma unroll
                    for (int r = 0; r < (1 << E1); ++r) tm_ld(tcol + r * 128, y[r]);
#pragma unroll
                    for (int j = 0; j < 16 / WGS; ++j) {
                        tm_wait(y[0]);
#pragma unroll
                        for (int r = 1; r < (1 << E1); ++r) tm_pin(y[r]);
                        u64 x[1 << E1];
                        combine<E1>(y, x);
                        if (j + 1 < 16 / WGS) {
#pragma unroll
                            for (int r = 0; r < (1 << E1); ++r) tm_ld(tcol + r * 128 + (j + 1) * 8, y[r]);
                        }
#pragma unroll
                        for (int s = 0; s < (1 << E1); ++s) {
                            const u32 aa = wgi * (16 / WGS) + j + 16 * s;
                            const u64 f = lds64(smT + 8 * ((aa << C::LR2) + (r2 << 4) + i2));
                            sts64(smD + op_addr<C::E2P>((aa << C::LW) + w, (i2 << C::E2P) | r2), mul_nc(x[s], f));
                        }
                    }
                }
                fence_async();
                tc_before();
                team_sync(team);
                if (tid == 0) {
                    tc_after();
#pragma unroll
                    for (int u = 0; u < C::UNITS2; ++u)
#pragma unroll
                        for (int r = 0; r < (1 << C::E2P); ++r)
                            mma_block(tmem + ((u << C::E2P) + r) * 128, smD + ((u << C::E2P) + r) * BLK, smB2 + r * BLK, 128);
                    mma_commit(bar);
                }
                ok = ok && mbar_wait(bar, phase);
                phase ^= 1;
                tc_after();
                if (t + TEAMS < t1) load(t + TEAMS);
                // Round 2 outputs b = b' + 16 s of row (a, w): output index a + R1 b of transform w.
#pragma unroll
                for (int u = 0; u < C::UNITS2; ++u) {
                    const u32 row = u * 128 + trow, w = row & (W - 1), aa = row >> C::LW;
                    const u32 tcol = tlane + (u << C::E2P) * 128 + wgi * (16 / WGS) * 8;
                    Limbs y[1 << C::E2P];
#pragma unroll
                    for (int r = 0; r < (1 << C::E2P); ++r) tm_ld(tcol + r * 128, y[r]);
                    u64* o;          // output (a, b = 0)
                    const u64* tp = nullptr;
                    u64 step;        // words between consecutive b
                    if constexpr (FIRST) {
                        const u32 rho = (t << C::LW) + w, plane = rho >> a.l2;
                        const u64 off = ((u64)(q + (aa << a.lE)) << a.l2) + (rho & (u32)(M2 - 1));
                        o = a.out + ((u64)plane << a.logN) + off;
                        tp = a.tab + off;
                        step = 1ull << (C::LR1 + a.lE + a.l2);
                    } else {
                        const u32 rho = (t << C::LW) + w, plane = rho >> lN1;
                        o = a.out + ((u64)plane << a.logN) + (rho & ((1u << lN1) - 1)) + ((u64)aa << lN1);
                        step = 1ull << (C::LR1 + lN1);
                    }
#pragma unroll
                    for (int j = 0; j < 16 / WGS; ++j) {
                        const u32 b0 = wgi * (16 / WGS) + j;
                        u64 f[1 << C::E2P];
                        if constexpr (FIRST) {
#pragma unroll
                            for (int s = 0; s < (1 << C::E2P); ++s)
                                f[s] = __ldg(reinterpret_cast<const unsigned long long*>(tp + (b0 + 16 * s) * step));
                        }
                        tm_wait(y[0]);
#pragma unroll
                        for (int r = 1; r < (1 << C::E2P); ++r) tm_pin(y[r]);
                        u64 x[1 << C::E2P];
                        combine<C::E2P>(y, x);
                        if (j + 1 < 16 / WGS) {
#pragma unroll
                            for (int r = 0; r < (1 << C::E2P); ++r) tm_ld(tcol + r * 128 + (j + 1) * 8, y[r]);
                        }
#pragma unroll
                        for (int s = 0; s < (1 << C::E2P); ++s)
                            o[(b0 + 16 * s) * step] = FIRST ? mul_nc(x[s], f[s]) : gl_canon(x[s]);
                    }
                }
            } else {
#pragma unroll
                for (int h = 0; h < C::HALVES; ++h) {
                    constexpr int NO = 16 / C::HALVES;  // outputs a' of a turn
                    if (h) {
                        tc_before();
                        team_sync(team);  // the turn's tensor memory has been read
                    }
                    if (tid == 0) {
                        tc_after();
#pragma unroll
                        for (int u = 0; u < C::UNITS1; ++u)
#pragma unroll
                            for (int r = 0; r < (1 << E1); ++r)
                                mma_block(tmem + ((u << E1) + r) * (8 * NO), smD + ((u << E1) + r) * BLK,
                                          smB1 + r * BLK + h * NO * 1024, 8 * NO);
                        mma_commit(bar);
                    }
                    ok = ok && mbar_wait(bar, phase);
                    phase ^= 1;
                    tc_after();
                    if (h + 1 == C::HALVES && t + TEAMS < t1) load(t + TEAMS);
#pragma unroll
                    for (int u = 0; u < C::UNITS1; ++u) {
                        const u32 rho = (t << C::LW) + u * 128 + trow;
                        const u32 tcol = tlane + (u << E1) * (8 * NO) + wgi * (NO / WGS) * 8;
                        Limbs y[1 << E1];
#pragma unroll
                        for (int r = 0; r < (1 << E1); ++r) tm_ld(tcol + r * (8 * NO), y[r]);
                        u64* o;
                        const u64* tp = nullptr;
                        u64 step;
                        if constexpr (FIRST) {
                            const u32 plane = rho >> a.l2;
                            const u64 off = ((u64)q << a.l2) + (rho & (u32)(M2 - 1));
                            o = a.out + ((u64)plane << a.logN) + off;
                            tp = a.tab + off;
                            step = 1ull << (a.lE + a.l2);
                        } else {
                            const u32 plane = rho >> lN1;
                            o = a.out + ((u64)plane << a.logN) + (rho & ((1u << lN1) - 1));
                            step = 1ull << lN1;
                        }
#pragma unroll
                        for (int j = 0; j < NO / WGS; ++j) {
                            const u32 a0 = h * NO + wgi * (NO / WGS) + j;
                            u64 f[1 << E1];
                            if constexpr (FIRST) {
#pragma unroll
                                for (int s = 0; s < (1 << E1); ++s)
                                    f[s] = __ldg(reinterpret_cast<const unsigned long long*>(tp + (a0 + 16 * s) * step));
                            }
                            tm_wait(y[0]);
#pragma unroll
                            for (int r = 1; r < (1 << E1); ++r) tm_pin(y[r]);
                            u64 x[1 << E1];
                            combine<E1>(y, x);
                            if (j + 1 < NO / WGS) {
#pragma unroll
                                for (int r = 0; r < (1 << E1); ++r) tm_ld(tcol + r * (8 * NO) + (j + 1) * 8, y[r]);
                            }
#pragma unroll
                            for (int s = 0; s < (1 << E1); ++s)
                                o[(a0 + 16 * s) * step] = FIRST ? mul_nc(x[s], f[s]) : gl_canon(x[s]);
                        }
                    }
                }
            }
        }
        cp_wait_all();
    }
    if (!ok && a.err) atomicOr_system(a.err, TX_ERR_TIMEOUT);
    tc_before();
    __syncthreads();
    if (threadIdx.x < 32) {
        tc_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(s_tmem), "n"(TEAMS * TEAM_COLS));
    }
}

typedef void (*Dft8Kernel)(Dft8Args);
struct Variant {
    Dft8Kernel k;
    u32 smem, log_rows;  // transforms of a tile
};
template <int E1, int E2, bool F>
Variant variant() { return Variant{k_dft8<E1, E2, F>, Cfg<E1, E2, F>::SMEM, (u32)Cfg<E1, E2, F>::LW}; }

// The pass kernel for `bits` index bits: one round of 4, 5 or 6 bits or two
// rounds of 4 + 4, 5 + 4 or 5 + 5.
template <bool F>
Variant pass_variant(u32 bits) {
    switch (bits) {
        case 4: return variant<0, -1, F>();
        case 5: return variant<1, -1, F>();
        case 6: return variant<2, -1, F>();
        case 8: return variant<0, 0, F>();
        case 9: return variant<1, 0, F>();
        case 10: return variant<1, 1, F>();
    }
    return Variant{nullptr, 0, 0};
}

}  // namespace

// Bits of the first and last pass for a message of 2^lm words per plane.
static bool dft8_split(u32 lm, u32* l1, u32* l2) {
    static const unsigned char first[21] = {0, 0, 0, 0, 0, 0, 0, 0, 4, 5, 5, 6, 6, 8, 8, 9, 10, 9, 9, 10, 10};
    if (lm < 8 || lm > 20) return false;
    *l1 = first[lm];
    *l2 = lm - first[lm];
    return true;
}

bool dft8_applicable(u32 logN, u32 logX, u32 planes) {
    u32 l1, l2;
    if (logN > TW_LOG || logX >= logN || !dft8_split(logN - logX, &l1, &l2)) return false;
    // whole tiles only
    const u64 r1 = (u64)planes << l2, r2 = (u64)planes << (logX + l1);
    return r1 >> 31 == 0 && r2 >> 31 == 0 && (r1 & ((1u << pass_variant<true>(l1).log_rows) - 1)) == 0 &&
           (r2 & ((1u << pass_variant<false>(l2).log_rows) - 1)) == 0;
}
u32 dft8_first_bits(u32 logN, u32 logX) {
    u32 l1, l2;
    return dft8_split(logN - logX, &l1, &l2) ? logX + l1 : 0;
}

int launch_dft8(const LdeArgs& L, u32 logX, cudaStream_t st) {
    u32 l1, l2;
    if (!dft8_split(L.logN - logX, &l1, &l2)) return -1;
    Dft8Args a{};
    for (int c = 0; c < 3; ++c) a.src[c] = L.src[c];
    a.in = L.tmp;
    a.depth = L.depth;
    a.logN = L.logN;
    a.lE = logX;
    a.l1 = l1;
    a.l2 = l2;
    a.tw_hi = L.tw_hi;
    a.tw_lo = L.tw_lo;
    a.err = L.err;
    const u32 sms = device_sms();
    const Variant f = pass_variant<true>(l1), g = pass_variant<false>(l2);
    a.out = L.tmp;
    a.tab = L.tables ? L.tables->get(L.logN, logX + l1) : nullptr;
    a.tiles_per_q = (u32)(((u64)L.planes << l2) >> f.log_rows);
    a.total = a.tiles_per_q << logX;
    f.k<<<std::min(sms, (a.total + 1) / 2), TEAMS * TT, f.smem, st>>>(a);
    a.out = L.out;
    a.tab = nullptr;
    a.tiles_per_q = a.total = (u32)(((u64)L.planes << (logX + l1)) >> g.log_rows);
    g.k<<<std::min(sms, (a.total + 1) / 2), TEAMS * TT, g.smem, st>>>(a);
    count_launches(2);
    return 0;
}

int dft8_prepare() {
    for (u32 b = 4; b <= 10; ++b)
        for (int f = 0; f < 2; ++f) {
            const Variant v = f ? pass_variant<true>(b) : pass_variant<false>(b);
            if (v.k && cudaFuncSetAttribute(v.k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)v.smem) != cudaSuccess)
                return -1;
        }
    return 0;
}

}  // namespace wg
