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
// What bounds it: the integer pipes again (45-55 instructions per output and
// round: join 13-20, factor 21, addresses and shared memory; ALU 65 %, FMA 55 %
// busy at 60 % issue), then HBM for the pass boundaries; the contraction itself
// takes 1/8 clock per output and SM, a fifth of the time, under the joins of the
// other tile.  Measured on B200 against the butterfly passes of k_ntt.cu: 16
// planes 2^20 -> 2^22 682 us against 1658 (four tiles' joins at 0.39 T outputs a
// second and round), 48 planes 2^16 -> 2^21 853 against 1846, 48 planes 2^12 ->
// 2^20 338 against 752.  Two independent halves of a CTA with a barrier after
// each round (8 warps each, cp.async copies of 8 bytes) took 872 / 1105 / 431;
// word-pair loads a round ahead instead of those copies were the larger part.
#include <algorithm>
#include <type_traits>

#include "gl.cuh"
#include "i8mma.cuh"
#include "launch.h"
#include "transcript.cuh"

namespace wg {

namespace {

constexpr int WARPS = 16;               // warps that join (all 128 rows, a quarter of the outputs per warpgroup)
constexpr int JT = 32 * WARPS;          // their threads; one more warp issues the contractions
constexpr int WGS = WARPS / 4;
constexpr int BATCH = 4;                // outputs joined at a time: their chains interleave, their loads go out together
constexpr u32 REGION = 256;             // tensor-memory columns of one of the two tiles in flight

// ---- joining the byte sums -------------------------------------------------
// u_j = l_(2j) + 2^8 l_(2j+1) <= 257 * 8323200 < 2^31: four digits of base 2^16.
struct U4 {
    u32 u[4];
};
__device__ __forceinline__ U4 join(const u32* l) {
    U4 r;
#pragma unroll
    for (int j = 0; j < 4; ++j) r.u[j] = l[2 * j] + (l[2 * j + 1] << 8);
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
__device__ __forceinline__ W2 u_w(const U4& a) { return W2{madw(a.u[1], 65536u, a.u[0]), madw(a.u[3], 65536u, a.u[2])}; }

// Digits of base 2^16 (u_2 < 2^32 - 2^16) as some 64-bit representative mod p.
// With h = u_3 >> 16 the part above 2^64 is h 2^64 = (2^32 - 1) h: h is added to
// u_2, then taken off (u_0, u_2 + h), which cannot borrow (h > 0 makes its upper
// half positive); the carry of one 64-bit addition is left to fold in.
__device__ __forceinline__ u64 u_reduce(const U4& a) {
    u64 s;
    asm("{\n\t.reg .u32 h, d, m, s1, x, c;\n\t.reg .u64 t;\n\t"
        "shr.u32 h, %4, 16;\n\t"
        "add.u32 m, %3, h;\n\t"
        "shl.b32 s1, %2, 16;\n\t"
        "prmt.b32 x, %2, %4, 0x5432;\n\t"  // u_1 >> 16 | u_3 << 16
        "sub.cc.u32 d, %1, h;\n\t"
        "subc.u32 m, m, 0;\n\t"
        "add.cc.u32 d, d, s1;\n\t"
        "addc.cc.u32 m, m, x;\n\t"
        "addc.u32 c, 0, 0;\n\t"
        "mov.b64 t, {d, m};\n\t"
        "mad.wide.u32 %0, c, 0xFFFFFFFF, t;\n\t}"  // after a carry m + x < 2^32 - 1: no second one
        : "=l"(s)
        : "r"(a.u[0]), "r"(a.u[1]), "r"(a.u[2]), "r"(a.u[3]));
    return s;
}
// a b mod p for any 64-bit a, b: some 64-bit representative.  Four 32 x 32
// products joined on one carry chain and reduced (2^64 = 2^32 - 1, 2^96 = -1).
__device__ __forceinline__ u64 mul_nc(u64 a, u64 b) {
    u64 s;
    asm("{\n\t.reg .u32 a0, a1, b0, b1, l0, l1, h0, h1, x0, x1, y0, y1, m;\n\t.reg .u64 p, q, r, t;\n\t"
        "mov.b64 {a0, a1}, %1;\n\t"
        "mov.b64 {b0, b1}, %2;\n\t"
        "mul.wide.u32 p, a0, b0;\n\t"
        "mul.wide.u32 q, a0, b1;\n\t"
        "mul.wide.u32 r, a1, b0;\n\t"
        "mul.wide.u32 t, a1, b1;\n\t"
        "mov.b64 {l0, l1}, p;\n\t"
        "mov.b64 {x0, x1}, q;\n\t"
        "mov.b64 {y0, y1}, r;\n\t"
        "mov.b64 {h0, h1}, t;\n\t"
        "add.cc.u32 l1, l1, x0;\n\t"
        "addc.cc.u32 h0, h0, x1;\n\t"
        "addc.u32 h1, h1, 0;\n\t"
        "add.cc.u32 l1, l1, y0;\n\t"
        "addc.cc.u32 h0, h0, y1;\n\t"
        "addc.u32 h1, h1, 0;\n\t"
        // minus h1; a borrow is 2^64 = 2^32 - 1 too much
        "sub.cc.u32 l0, l0, h1;\n\t"
        "subc.cc.u32 l1, l1, 0;\n\t"
        "subc.u32 m, 0, 0;\n\t"
        "sub.cc.u32 l0, l0, m;\n\t"
        "subc.u32 l1, l1, 0;\n\t"
        // plus h0 (2^32 - 1); a carry is 2^32 - 1 too little, and adding that cannot carry again
        "mul.wide.u32 p, h0, 0xFFFFFFFF;\n\t"
        "mov.b64 {x0, x1}, p;\n\t"
        "add.cc.u32 l0, l0, x0;\n\t"
        "addc.cc.u32 l1, l1, x1;\n\t"
        "addc.u32 m, 0, 0;\n\t"
        "sub.u32 m, 0, m;\n\t"
        "add.cc.u32 l0, l0, m;\n\t"
        "addc.u32 l1, l1, 0;\n\t"
        "mov.b64 %0, {l0, l1};\n\t}"
        : "=l"(s)
        : "l"(a), "l"(b));
    return s;
}

// The outputs X[a + 16 s], s < 2^E, from the blocks' sums for output a (the
// k-th of the loaded ones).
template <int E, int NB>
__device__ __forceinline__ void combine(const Limbs<NB> (&y)[1 << E], int k, u64* x) {
    if constexpr (E == 0) {
        x[0] = u_reduce(join(y[0].l + 8 * k));
    } else if constexpr (E == 1) {
        const U4 a = join(y[0].l + 8 * k), b = join(y[1].l + 8 * k);
        x[0] = u_reduce(u_add(a, b));
        x[1] = u_reduce(u_sub(a, b));
    } else {
        const U4 a = join(y[0].l + 8 * k), b = join(y[1].l + 8 * k), c = join(y[2].l + 8 * k), d = join(y[3].l + 8 * k);
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
__device__ __forceinline__ void build_b(unsigned char* smB, u32 q, u32 lE, const u64* hi, const u64* lo) {
    for (u32 k = threadIdx.x; k < (256u << E); k += JT) {
        const u32 i = k & 15, a = (k >> 4) & 15, r = k >> 8;
        const u64 v = root_pow((u64)((i << E) + r) * (q + ((u64)a << lE)), 4 + E + lE, hi, lo);
        expand_bytes(v, smB + r * BLK + a * 1024, i);
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
    static constexpr int LT = !TWO && E1 == 2 ? 13 : 12;  // words of a tile
    static constexpr int LW = LT - L;                     // transforms of a tile
    static constexpr int UNITS1 = 1 << (LT - 7 - LR1);    // 128-row groups of round 1
    static constexpr int UNITS2 = 1 << (LT - 7 - LR2);
    static constexpr int HALVES = !TWO && E1 == 2 ? 2 : 1;  // outputs of a round in two turns of tensor memory
    static constexpr u32 DATA = 8u << LT;
    // Rows of round 1 are permuted by this (XOR on the index mod 16), so that
    // the word pairs of neighbouring transforms differ mod 8.
    static __device__ __forceinline__ u32 swz(u32 w) { return ((w >> 1) << (E1 + E2P)) & 7; }
    static constexpr int NL = (1 << LT) / JT / 2;  // word pairs of a tile per thread
    static constexpr u32 B1 = BLK << E1, B2 = TWO ? BLK << E2P : 0, TWB = TWO ? 8u << L : 0;
    static constexpr u32 SMEM = 2 * DATA + B1 + B2 + TWB + 1024;
};

// Where the outputs of a round go: word k of this thread's row at base + k step
// bytes (and its factor at tab + k step).
struct Dest {
    char* o;
    const char* tp;
    u32 step;
};
// Output a of batch entry k: a' = k >> E, plus 16 s.
template <int E>
__device__ __forceinline__ constexpr u32 out_of(int k) { return (u32)((k >> E) + 16 * (k & ((1 << E) - 1))); }

template <int E>
struct Batch {  // the byte sums of BATCH outputs
    Limbs<(BATCH >> E)> y[1 << E];
    __device__ __forceinline__ void load(u32 col, u32 rs) {  // rs: columns per block
#pragma unroll
        for (int r = 0; r < (1 << E); ++r) tm_ld(col + r * rs, y[r]);
    }
    __device__ __forceinline__ void join_all(u64 (&x)[BATCH]) {  // after the wait
        tm_wait();
#pragma unroll
        for (int r = 0; r < (1 << E); ++r) tm_pin(y[r]);
#pragma unroll
        for (int k = 0; k < (BATCH >> E); ++k) combine<E>(y, k, x + (k << E));
    }
};
template <int E>
__device__ __forceinline__ void factors(u64 (&f)[BATCH], const Dest& d, u32 a0) {
    const char* p = d.tp + (u64)d.step * a0;
#pragma unroll
    for (int k = 0; k < BATCH; ++k) f[k] = __ldg(reinterpret_cast<const unsigned long long*>(p + (u64)d.step * out_of<E>(k)));
}
template <int E, bool FACTOR>
__device__ __forceinline__ void finish(u64 (&x)[BATCH], const u64 (&f)[BATCH], const Dest& d, u32 a0) {
    char* p = d.o + (u64)d.step * a0;
#pragma unroll
    for (int k = 0; k < BATCH; ++k) x[k] = FACTOR ? mul_nc(x[k], f[k]) : gl_canon(x[k]);
#pragma unroll
    for (int k = 0; k < BATCH; ++k) *reinterpret_cast<u64*>(p + (u64)d.step * out_of<E>(k)) = x[k];
}

// Two tiles are in flight, each with its own shared-memory buffer and half of
// the tensor memory: while the contraction of one runs (or its copies are under
// way) all 16 warps join the other.  Barrier full[b]: tile b's operand is in
// place and its tensor memory read (one arrival per warp); done[b]: its
// contraction has finished.  The joining warps never wait for one another.
template <int E1, int E2, bool FIRST>
__global__ void __launch_bounds__(JT + 32, 1) k_dft8(const __grid_constant__ Dft8Args a) {
    using C = Cfg<E1, E2, FIRST>;
    constexpr int G1 = BATCH >> E1;
    extern __shared__ unsigned char smem_raw[];
    __shared__ u32 s_tmem;
    __shared__ __align__(8) u64 s_bar[5];
    const u32 base = (smem_u32(smem_raw) + 1023) & ~1023u;
    unsigned char* const gbase = smem_raw + (base - smem_u32(smem_raw));
    const u32 tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const bool issuer = warp == WARPS;
    unsigned char* const gB = gbase + 2 * C::DATA;
    u64* const gT = reinterpret_cast<u64*>(gB + C::B1 + C::B2);
    const u32 smB1 = base + 2 * C::DATA, smB2 = smB1 + C::B1;
    const u32 full = smem_u32(&s_bar[0]), done = smem_u32(&s_bar[2]);  // [b] at + 8 b
    const u32 drain = smem_u32(&s_bar[4]);

    if (issuer) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "n"(2 * REGION)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        for (u32 b = 0; b < 2; ++b) {
            mbar_init(full + 8 * b, WARPS);
            mbar_init(done + 8 * b, 1);
        }
        mbar_init(drain, 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    tc_before();
    __syncthreads();
    tc_after();
    const u32 tmem = s_tmem;
    const u32 tlane = tmem + ((warp & 3) << 21);  // this warp's 32 rows
    const u32 wgi = warp >> 2;
    const u32 trow = ((warp & 3) << 5) | lane;
    u32 ph0 = 0, ph1 = 0;  // phases of full[b] (issuer) or done[b] (joining warps)
    bool ok = true;

    const u64 M2 = 1ull << a.l2;
    const u32 lN1 = a.logN - a.l2;  // 2^lE M1
    constexpr u32 W = 1u << C::LW;

    auto await = [&](u32 bar, u32 b) {
        u32& ph = b ? ph1 : ph0;
        ok = ok && mbar_wait(bar + 8 * b, ph);
        ph ^= 1;
        tc_after();
    };
    // This warp's part of tile b's operand is in place, and it has read the tile's tensor memory.
    auto ready = [&](u32 b) {
        fence_async();
        tc_before();
        __syncwarp();
        if (lane == 0 && ok) mbar_arrive(full + 8 * b);  // after a wait that ran out nothing is handed on
    };

    // ---- a tile's loads: word pairs adjacent in memory, one round ahead -------
    // A thread's pair j differs from its pair 0 by constants: g_step(j) words of
    // memory, and s_of(j) in shared memory.  The lanes are chosen so that each
    // half-warp's stores (8 bytes a lane) fall on distinct banks.
    ulonglong2 pre[C::NL];
    u32 g0 = 0, s0 = 0, row0 = 0;  // word offset in the tile's block of memory, byte offset in the buffer, row
    if (!issuer) {
        const u32 x = tid;
        u32 d = 0;
        if constexpr (C::TWO) {
            u32 w, i2, r2, i1, r1;
            if constexpr (FIRST) {  // pair: transforms w, w + 1; j: high bits of d
                constexpr int Z = E1 + C::E2P + 1;  // low bits of i2 in the lane
                w = (x & (W / 2 - 1)) * 2;
                u32 y = x >> (C::LW - 1);
                i1 = y & 1;
                i2 = (y >> 1) & ((1u << Z) - 1);
                y >>= Z + 1;
                i2 |= (y & ((1u << (4 - Z)) - 1)) << Z;
                y >>= 4 - Z;
                r2 = y & ((1u << C::E2P) - 1);
                i1 |= (y >> C::E2P) << 1;
                r1 = 0;
            } else {  // pair: columns d2, d2 + 1; j: high bits of w
                constexpr int D = 2 + C::E2P;  // bits 1 .. D of d2, low bits of i1, bit D + 1 of d2
                constexpr int I = 2 - C::E2P;
                u32 e2 = (x & ((1u << D) - 1)) * 2;
                u32 y = x >> D;
                i1 = y & ((1u << I) - 1);
                y >>= I;
                e2 |= (y & 1) << (D + 1);
                y >>= 1;
                i1 |= (y & ((1u << (4 - I)) - 1)) << I;
                y >>= 4 - I;
                r1 = y & ((1u << E1) - 1);
                w = y >> E1;
                r2 = e2 & ((1u << C::E2P) - 1);
                i2 = e2 >> C::E2P;
            }
            d = (i1 << E1) | r1;
            const u32 d2 = (i2 << C::E2P) | r2;
            // row of (d2, w): the 16 words i2 of one block row of round 2 in 16 lanes
            row0 = (((r2 << C::LW) | w) << 4) | (i2 ^ C::swz(w));
            g0 = FIRST ? ((d2 + (d << C::LR2)) << a.l2) + w : (w << a.l2) + d2 + (d << C::LR2);
        } else if constexpr (FIRST) {  // pair: rows, rows + 1; j: high bits of d
            row0 = (x & 3) * 2;
            u32 y = x >> 2;
            u32 i = y & 3;
            y >>= 2;
            row0 |= (y & ((W >> 3) - 1)) << 3;
            i |= (y >> (C::LW - 3)) << 2;
            d = i << E1;
            g0 = d << a.l2;
        } else {  // pair: words d, d + 1 of a row; j: high bits of the row
            d = (x & (8 * (1u << E1) - 1)) * 2;
            row0 = x >> (3 + E1);
            g0 = (row0 << C::LR1) + d;
        }
        s0 = op_addr<E1>(row0, d);
    }
    auto g_step = [&](int j) -> u32 {  // words
        if constexpr (FIRST) {
            const u32 d = E1 == 0 ? j << 2 : E1 == 1 ? ((j & 1) << 4) | j >> 1 : ((j & 1) << 5) | j >> 1;
            return (d << (C::TWO ? C::LR2 : 0)) << a.l2;
        } else {
            return C::TWO ? (u32)(j * (W / C::NL)) << a.l2 : (u32)(j * (W / C::NL)) << C::LR1;
        }
    };
    auto s_of = [&](int j) -> u32 {
        if constexpr (FIRST) {  // bits 2, 3 of the word index in its block move 16-byte chunks 1, 2; the block follows
            if constexpr (E1 == 0) return s0 ^ ((u32)j << 5);
            return (s0 ^ ((u32)(j & 1) << 6)) + (u32)(j >> 1) * BLK;
        } else if constexpr (C::TWO) {  // w moves 16-row groups and the permutation
            const u32 w = j * (W / C::NL);
            return (s0 ^ (C::swz(w) << 7 | C::swz(w) << 4)) + w * 16 * 128;
        } else {
            return s0 + j * (W / C::NL) * 128;
        }
    };
    auto fetch = [&](u32 t) {
        const u32 rho = t << C::LW;
        const u64* p;
        if constexpr (FIRST) {
            const u32 plane = (rho >> a.l2) + (C::TWO ? 0 : row0 >> a.l2);
            const u32 comp = (plane >= a.depth) + (plane >= 2 * a.depth);
            const u64* m = comp == 0 ? a.src[0] : comp == 1 ? a.src[1] : a.src[2];
            p = m + ((u64)(plane - comp * a.depth) << (a.l1 + a.l2)) + (rho & (u32)(M2 - 1)) + g0 +
                (C::TWO ? 0 : row0 & (u32)(M2 - 1));
        } else {
            p = a.in + ((u64)rho << a.l2) + g0;
        }
#pragma unroll
        for (int j = 0; j < C::NL; ++j) pre[j] = __ldg(reinterpret_cast<const ulonglong2*>(p + g_step(j)));
    };
    auto put = [&](u32 b) {
        unsigned char* const sm = gbase + b * C::DATA;
#pragma unroll
        for (int j = 0; j < C::NL; ++j) {
            const u32 o = s_of(j);
            if constexpr (!C::TWO && !FIRST && E1 == 0) {  // both words in one 16-byte chunk
                *reinterpret_cast<ulonglong2*>(sm + o) = pre[j];
            } else {
                *reinterpret_cast<u64*>(sm + o) = pre[j].x;
                u32 o2;
                if constexpr (C::TWO && FIRST) o2 = o + 16 * 128;                         // w + 1
                else if constexpr (C::TWO && C::E2P == 1) o2 = o + ((16 * 128) << C::LW);  // the other residue of d2
                else if constexpr (C::TWO || FIRST) o2 = o ^ (128 | 16);                   // the next row
                else o2 = o + BLK;                                                         // the next block
                *reinterpret_cast<u64*>(sm + o2) = pre[j].y;
            }
        }
    };
    // Every round is two batches a thread; the second one's sums (and factors)
    // are loaded while the first is multiplied and stored.
    //
    // Round 1 of a two-round pass: outputs a = a' + 16 s of row (d2, w), times
    // the factor, to word d2 of row (a, w) of buffer b.
    auto round1 = [&](u32 b) {
        await(done, b);
        constexpr u32 AW = 16 / WGS;
        unsigned char* const sm = gbase + b * C::DATA;
        Batch<E1> y;
        u64 f[BATCH], x[BATCH];
        const u32 tcol = tlane + b * REGION + wgi * AW * 8;
        constexpr u32 NEXT = C::UNITS1 == 2 ? 128 << E1 : G1 * 8;
        y.load(tcol, 128);
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int u = C::UNITS1 == 2 ? k : 0;
            const u32 ak = C::UNITS1 == 2 ? 0 : k * G1;  // outputs wgi AW + ak ..
            const u32 row = u * 128 + trow, hi = row >> 4, w = hi & (W - 1), r2 = hi >> C::LW;
            const u32 i2 = (row & 15) ^ C::swz(w);
            const u64* ft = gT + ((wgi * AW) << C::LR2) + (r2 << 4) + i2;
            const u32 o0 = op_addr<C::E2P>(((wgi * AW) << C::LW) + w, (i2 << C::E2P) | r2);
#pragma unroll
            for (int k2 = 0; k2 < BATCH; ++k2) f[k2] = ft[(ak + out_of<E1>(k2)) << C::LR2];
            y.join_all(x);
            if (k == 0) y.load(tcol + NEXT, 128);
#pragma unroll
            for (int k2 = 0; k2 < BATCH; ++k2) x[k2] = mul_nc(x[k2], f[k2]);
#pragma unroll
            for (int k2 = 0; k2 < BATCH; ++k2) {
                const u32 da = ak + out_of<E1>(k2);  // row (a, w) is W da rows on
                const u32 o = (W == 4 && (da & 1) ? o0 ^ 64 : o0) + da * W * 128;
                *reinterpret_cast<u64*>(sm + o) = x[k2];
            }
        }
    };
    // The last round of the pass (radix 2^(4 + E)): dest(u) gives the words of
    // this thread's row of unit u; `before` runs once the contraction is done.
    auto last_round = [&](auto ec, u32 b, u32 a_first, auto dest, auto before) {
        constexpr int E = decltype(ec)::value;
        constexpr int G = BATCH >> E, UNITS = C::TWO ? C::UNITS2 : C::UNITS1, NO = 16 / C::HALVES;
        constexpr u32 RS = 8 * NO, NEXT = UNITS == 2 ? RS << E : G * 8;
        const u32 c0 = wgi * (NO / WGS);
        const Dest d0 = dest(0), d1 = UNITS == 2 ? dest(1) : d0;
        const u32 a0 = a_first + c0, a1 = UNITS == 2 ? a0 : a0 + G;
        u64 f0[BATCH], f1[BATCH], x[BATCH];
        if constexpr (FIRST) factors<E>(f0, d0, a0);
        await(done, b);
        before();
        Batch<E> y;
        const u32 tcol = tlane + b * REGION + c0 * 8;
        y.load(tcol, RS);
        if constexpr (FIRST) factors<E>(f1, d1, a1);
        y.join_all(x);
        y.load(tcol + NEXT, RS);
        finish<E, FIRST>(x, f0, d0, a0);
        y.join_all(x);
        finish<E, FIRST>(x, f1, d1, a1);
    };
    // Round 2 of tile t: output b of row (a, w) is output index a + R1 b of transform w.
    auto round2 = [&](u32 t, u32 b, u32 q, auto before) {
        const u32 rho = t << C::LW;  // the tile's part of an address is the same in all threads
        auto dest = [&](int u) {
            const u32 row = u * 128 + trow, w = row & (W - 1), aa = row >> C::LW;
            Dest d{};
            if constexpr (FIRST) {
                const u64 off = ((u64)q << a.l2) + (rho & (u32)(M2 - 1)), own = ((u64)aa << (a.lE + a.l2)) + w;
                d.o = reinterpret_cast<char*>(a.out + (((u64)(rho >> a.l2) << a.logN) + off) + own);
                d.tp = reinterpret_cast<const char*>(a.tab + off + own);
                d.step = 8u << (C::LR1 + a.lE + a.l2);
            } else {
                d.o = reinterpret_cast<char*>(a.out + (((u64)(rho >> lN1) << a.logN) + (rho & ((1u << lN1) - 1))) + (((u64)aa << lN1) + w));
                d.step = 8u << (C::LR1 + lN1);
            }
            return d;
        };
        last_round(std::integral_constant<int, C::E2P>{}, b, 0, dest, before);
    };
    // The round of a one-round pass on region b: turn b of tile t's outputs
    // (radix 64), or all of them.
    auto round0 = [&](u32 t, u32 b, u32 q, auto before) {
        const u32 rho = t << C::LW;
        auto dest = [&](int u) {
            const u32 row = u * 128 + trow;
            Dest d{};
            if constexpr (FIRST) {
                const u64 off = ((u64)q << a.l2) + (rho & (u32)(M2 - 1));
                const u32 own = row & (u32)(M2 - 1);
                d.o = reinterpret_cast<char*>(a.out + (((u64)(rho >> a.l2) << a.logN) + off) + (((u64)(row >> a.l2) << a.logN) + own));
                d.tp = reinterpret_cast<const char*>(a.tab + off + own);
                d.step = 8u << (a.lE + a.l2);
            } else {
                const u32 m = (1u << lN1) - 1;
                d.o = reinterpret_cast<char*>(a.out + (((u64)(rho >> lN1) << a.logN) + (rho & m)) + (((u64)(row >> lN1) << a.logN) + (row & m)));
                d.step = 8u << lN1;
            }
            return d;
        };
        last_round(std::integral_constant<int, E1>{}, b, C::HALVES == 2 ? b * (16 / C::HALVES) : 0, dest, before);
    };
    // The issuer's contractions of region b (none after a wait that ran out: their
    // operand may still be written).
    auto contract = [&](u32 b, u32 buf, bool second) {
        await(full, b);
        if (lane != 0 || !ok) return;
        const u32 smD = base + buf * C::DATA, d = tmem + b * REGION;
        constexpr int NO = 16 / C::HALVES;
        if (!second) {
#pragma unroll
            for (int k = 0; k < (C::UNITS1 << E1); ++k)
                mma_block(d + k * (8 * NO), smD + k * BLK, smB1 + (k & ((1 << E1) - 1)) * BLK + (C::HALVES == 2 ? b * NO * 1024 : 0),
                          8 * NO);
        } else {
#pragma unroll
            for (int k = 0; k < (C::UNITS2 << C::E2P); ++k)
                mma_block(d + k * 128, smD + k * BLK, smB2 + (k & ((1 << C::E2P) - 1)) * BLK, 128);
        }
        mma_commit(done + 8 * b);
    };

    const u32 lo_t = (u32)((u64)a.total * blockIdx.x / gridDim.x), hi_t = (u32)((u64)a.total * (blockIdx.x + 1) / gridDim.x);
    for (u32 cur = lo_t; cur < hi_t;) {
        const u32 q = FIRST ? cur / a.tiles_per_q : 0;
        const u32 t0 = cur - q * a.tiles_per_q;
        const u32 cnt = min(hi_t - cur, a.tiles_per_q - t0);
        cur += cnt;
        // Every contraction of the previous coset is done (its last round has
        // been read); a wait that ran out ends the CTA here.
        if (__syncthreads_or(!ok)) break;
        if (!issuer) {
            fetch(t0);
            const u32 lEq = FIRST ? a.lE : 0;
            build_b<E1>(gB, q, lEq, a.tw_hi, a.tw_lo);
            if constexpr (C::TWO) {
                build_b<E2>(gB + C::B1, 0, 0, a.tw_hi, a.tw_lo);
                // inter-round factors w_{2^(L + lE)}^(d2 (q + 2^lE a)) at [a][r2][i2]
                for (u32 k = tid; k < (1u << C::L); k += JT) {
                    const u32 i2 = k & 15, r2 = (k >> 4) & ((1u << C::E2P) - 1), aa = k >> C::LR2;
                    const u32 d2 = (i2 << C::E2P) | r2;
                    gT[k] = root_pow((u64)d2 * (q + ((u64)aa << lEq)), C::L + lEq, a.tw_hi, a.tw_lo);
                }
            }
            put(0);
            if (cnt > 1) {
                fetch(t0 + 1);
                put(1);
            }
        }
        fence_async();
        __syncthreads();
        if (issuer) {
            if constexpr (C::TWO) {
                for (u32 i = 0; i < cnt; i += 2) {
                    const bool two = i + 1 < cnt;
                    contract(0, 0, false);
                    if (two) contract(1, 1, false);
                    contract(0, 0, true);
                    if (two) contract(1, 1, true);
                }
            } else if constexpr (C::HALVES == 2) {
                for (u32 i = 0; i < cnt; ++i) {
                    contract(0, i & 1, false);
                    contract(1, i & 1, false);
                }
            } else {
                for (u32 i = 0; i < cnt; ++i) contract(i & 1, i & 1, false);
            }
        } else if constexpr (C::TWO) {
            ready(0);
            if (cnt > 1) ready(1);
            for (u32 i = 0; i < cnt; i += 2) {
                const u32 t = t0 + i;
                round1(0);
                ready(0);
                if (i + 2 < cnt) fetch(t + 2);
                if (i + 1 < cnt) {
                    round1(1);
                    ready(1);
                }
                round2(t, 0, q, [&] {
                    if (i + 2 < cnt) put(0);
                    if (i + 3 < cnt) fetch(t + 3);
                });
                if (i + 2 < cnt) ready(0);
                if (i + 1 < cnt) {
                    round2(t + 1, 1, q, [&] {
                        if (i + 3 < cnt) put(1);
                    });
                    if (i + 3 < cnt) ready(1);
                }
            }
        } else if constexpr (C::HALVES == 2) {
            ready(0);
            ready(1);
            for (u32 i = 0; i < cnt; ++i) {
                const u32 t = t0 + i;
                round0(t, 0, q, [&] {
                    if (i + 2 < cnt) fetch(t + 2);
                });
                if (i + 1 < cnt) ready(0);
                round0(t, 1, q, [&] {
                    if (i + 2 < cnt) put(i & 1);
                });
                if (i + 1 < cnt) ready(1);
            }
        } else {
            ready(0);
            if (cnt > 1) ready(1);
            if (cnt > 2) fetch(t0 + 2);
            for (u32 i = 0; i < cnt; ++i) {
                const u32 t = t0 + i, b = i & 1;
                round0(t, b, q, [&] {
                    if (i + 2 < cnt) put(b);
                    if (i + 3 < cnt) fetch(t + 3);
                });
                if (i + 2 < cnt) ready(b);
            }
        }
    }
    if (!ok && a.err) atomicOr_system(a.err, TX_ERR_TIMEOUT);
    tc_before();
    const bool failed = __syncthreads_or(!ok);
    if (issuer) {
        if (failed && lane == 0) {  // the contractions under way end before their memory goes
            mma_commit(drain);
            mbar_wait(drain, 0);
        }
        __syncwarp();
        tc_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(2 * REGION));
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
    f.k<<<std::min(sms, a.total), JT + 32, f.smem, st>>>(a);
    a.out = L.out;
    a.tab = nullptr;
    a.tiles_per_q = a.total = (u32)(((u64)L.planes << (logX + l1)) >> g.log_rows);
    g.k<<<std::min(sms, a.total), JT + 32, g.smem, st>>>(a);
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
