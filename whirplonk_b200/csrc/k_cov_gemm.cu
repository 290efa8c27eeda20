// k_cov_gemm.cu -- the STIR covector update of a large vector as an exact 8-bit
// contraction on the tensor cores.
//
//     cov[h 2^LO + l] += sum_j T_j[h] z_j^l,   T_j[h] = rlc_j z_j^(h 2^LO)
// (whir_prover.hpp:336-345, utilities.hpp:261-307) is, per component c of the
// target field, a matrix product over the points j: rows (c, h), columns l.
// The words T_j[h] are their own byte operand (A, K = 8 bytes of each point);
// z_j^l is expanded to the bytes of z_j^l 2^(8b) mod p in eight rows (B), so
// tcgen05.mma kind::i8 returns eight byte sums per element, which are joined,
// reduced and added to the covector once.  A point of the extension field (an
// out-of-domain sample) is three points over the components of z_j^l, its row
// entries those of the multiplication by T_j[h].
//
// Bound: 64 byte products per word product -- 3 2^20 elements x 200 points are
// 40 G, 18 us -- and 64 KB of operands per 1024 clocks and SM from L2.  The
// 192-bit multiply-accumulates of k_cov_accumulate run at 1.3 T word products a
// second.  Measured on B200, all covector updates of a proof (tables included):
// n = 24 rate 1/4 425 -> 152 us, n = 20 rate 1/8 100 -> 88, n = 18 rate 1/2 121
// -> 70.
//
// The operand images lie in the workspace's LDE scratch, which is free between
// commitments.  Where that is smaller -- folding 1 at rate 1/2: 190 words a row at
// 2^15 elements want 2.75 MB, and there are 1.5 -- the update runs from tables
// (k_cov_accumulate), as it does for vectors whose planes do not start at 16 bytes.
#include <algorithm>

#include "gl.cuh"
#include "i8mma.cuh"
#include "launch.h"
#include "state.cuh"

namespace wg {

namespace {

constexpr u32 CG_TILE_N = 256;      // columns of tensor memory per row tile: 32 elements l
constexpr u32 CG_STAGES = 3;
constexpr u32 CG_STAGE = 4 * BLK;   // two row tiles, one column tile of two blocks
constexpr u32 CG_SMEM = CG_STAGES * CG_STAGE + 1024;
constexpr int CG_EPI_WARPS = 8;     // warps 0..7 join, 8 copies, 9 issues

struct CovGemmArgs {
    u64* cov[3];
    u32 log_lo, log_hi;
    u32 rows, chunks;   // 3 2^log_hi, K blocks of 16 words
    const unsigned char* A;  // [row tile][chunk] operand blocks
    const unsigned char* B;  // [column tile][chunk] pairs of operand blocks
    u32* err;
};

// Word k of the contraction (a point, or a component of an Ext3 point) for the
// operand images; words past the last point are zero.
__global__ void __launch_bounds__(256) k_cov_gemm_tables(const ProofScalars* sc, int n_ext, int n_base, u32 log_lo, u32 log_hi,
                                                         u32 chunks, unsigned char* A, unsigned char* B, bool ext2) {
    const u32 K = chunks * 16, kw = 3 * n_ext + n_base;
    const u32 na = K << log_hi, nb = K << log_lo;
    for (u32 e = blockIdx.x * blockDim.x + threadIdx.x; e < na + nb; e += gridDim.x * blockDim.x) {
        const bool isA = e < na;
        const u32 x = isA ? e : e - na;
        const u32 lg = isA ? log_hi : log_lo;
        const u32 k = x >> lg, p = x & ((1u << lg) - 1);  // word, h or l
        const u64 ex = isA ? (u64)p << log_lo : p;
        E3 v = e3_zero();  // A: the row entries of components 0..2; B: c0
        if (k < kw) {
            const bool ext = k < 3 * (u32)n_ext;
            const u32 j = ext ? k / 3 : k - 2 * n_ext, s = ext ? k % 3 : 0;
            const E3 z = sc->stir_pts[j];
            if (!ext) {
                const u64 w = gl_pow(z.c0, ex);
                v = isA ? e3_mul_base(sc->stir_rlc[j], w) : e3_base(w);
            } else {
                const E3 w = ef_pow(z, ex, ext2);
                if (!isA) {
                    v.c0 = s == 0 ? w.c0 : s == 1 ? w.c1 : w.c2;
                } else {
                    const E3 t = ef_mul(sc->stir_rlc[j], w, ext2);
                    // column s of the multiplication by t: X^3 = 2, or X^2 = 7
                    const u64 t1d = ext2 ? gl_mul(t.c1, GL_EXT2_NR) : gl_add(t.c1, t.c1), t2d = gl_add(t.c2, t.c2);
                    if (s == 0) v = t;
                    else if (s == 1) v = ext2 ? E3{t1d, t.c0, 0} : E3{t2d, t.c0, t.c1};
                    else v = ext2 ? e3_zero() : E3{t1d, t2d, t.c0};
                }
            }
        }
        const u32 c = k >> 4, i = k & 15;
        if (isA) {
#pragma unroll
            for (u32 q = 0; q < 3; ++q) {
                const u32 row = (q << log_hi) + p, r = row & 127;
                *reinterpret_cast<u64*>(A + ((u64)(row >> 7) * chunks + c) * BLK + r * 128 + (((i >> 1) ^ (r & 7)) << 4) + (i & 1) * 8) =
                    q == 0 ? v.c0 : q == 1 ? v.c1 : v.c2;
            }
        } else {
            expand_bytes(v.c0, B + ((u64)(p >> 5) * chunks + c) * 2 * BLK + (p & 31) * 1024, i);
        }
    }
}

// Eight byte sums below 2^30 as one word mod p, canonical.
__device__ __forceinline__ u64 join_wide(const u32* l) {
    const u64 a = madw(l[1], 256u, l[0]), b = madw(l[3], 256u, l[2]), c = madw(l[5], 256u, l[4]), d = madw(l[7], 256u, l[6]);
    return gl_canon(w_reduce(W2{a + (b << 16), c + (d << 16)}));
}

// Two row tiles by one column tile per CTA: one warp copies operand blocks to a
// ring (bulk copies), one issues the contractions, and eight join at the end
// (all of tensor memory holds the two tiles' sums).
__global__ void __launch_bounds__(32 * (CG_EPI_WARPS + 2), 1) k_cov_gemm(const __grid_constant__ CovGemmArgs a) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ u32 s_tmem;
    __shared__ __align__(8) u64 bars[2 * CG_STAGES + 1];
    const u32 base = (smem_u32(smem_raw) + 1023) & ~1023u;
    const u32 warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const u32 full = smem_u32(bars), empty = full + 8 * CG_STAGES, done = empty + 8 * CG_STAGES;
    const u32 mt = blockIdx.y * 2, tiles = (a.rows + 127) / 128;
    const bool two = mt + 1 < tiles;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&s_tmem)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (threadIdx.x == 0)
        for (u32 s = 0; s < 2 * CG_STAGES + 1; ++s) mbar_init(full + 8 * s, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    tc_before();
    __syncthreads();
    tc_after();
    const u32 tmem = s_tmem;
    bool ok = true;
    if (warp == CG_EPI_WARPS) {
        if (lane == 0) {
            auto copy = [&](u32 dst, const unsigned char* src, u32 bytes, u32 bar) {
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                             "l"(src), "r"(bytes), "r"(bar)
                             : "memory");
            };
            u32 s = 0, ph = 0, armed = 0;
            for (u32 c = 0; c < a.chunks; ++c) {
                ok = mbar_wait(empty + 8 * s, ph ^ 1);
                if (!ok) break;
                const u32 bytes = (two ? 4 : 3) * BLK;
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(full + 8 * s), "r"(bytes) : "memory");
                const u32 st = base + s * CG_STAGE;
                copy(st, a.A + ((u64)mt * a.chunks + c) * BLK, BLK, full + 8 * s);
                if (two) copy(st + BLK, a.A + ((u64)(mt + 1) * a.chunks + c) * BLK, BLK, full + 8 * s);
                copy(st + 2 * BLK, a.B + ((u64)blockIdx.x * a.chunks + c) * 2 * BLK, 2 * BLK, full + 8 * s);
                armed = min(armed + 1, CG_STAGES);
                if (++s == CG_STAGES) s = 0, ph ^= 1;
            }
            ok = ring_drain(full, CG_STAGES, s, ph, armed) && ok;
        }
    } else if (warp == CG_EPI_WARPS + 1) {
        if (lane == 0) {
            u32 s = 0, ph = 0;
            for (u32 c = 0; c < a.chunks; ++c) {
                ok = mbar_wait(full + 8 * s, ph);
                if (!ok) break;
                tc_after();
                const u32 st = base + s * CG_STAGE;
                const u64 db = op_desc(st + 2 * BLK);
                for (u32 t = 0; t < (two ? 2u : 1u); ++t) {
                    const u64 da = op_desc(st + t * BLK);
#pragma unroll
                    for (u32 k = 0; k < 4; ++k) mma_i8(tmem + t * CG_TILE_N, da + 2 * k, db + 2 * k, op_idesc(CG_TILE_N), c | k);
                }
                mma_commit(empty + 8 * s);
                if (++s == CG_STAGES) s = 0, ph ^= 1;
            }
            mma_commit(done);
            ok = mbar_wait(done, 0) && ok;  // the contractions end before their memory goes
        }
    } else {
        ok = mbar_wait(done, 0);
        tc_after();
        const u32 t = warp >> 2, row = (mt + t) * 128 + (warp & 3) * 32 + lane;
        if (t == 0 || two) {  // (uniform in the warp)
            const u32 H = 1u << a.log_hi, comp = row >> a.log_hi;
            u64* p = comp == 0 ? a.cov[0] : comp == 1 ? a.cov[1] : a.cov[2];
            p += ((u64)(row & (H - 1)) << a.log_lo) + blockIdx.x * 32;
            const u32 col = tmem + t * CG_TILE_N + ((warp & 3) << 21);
#pragma unroll 1
            for (u32 l = 0; l < 32; l += 4) {
                Limbs<4> y;
                tm_ld(col + l * 8, y);
                ulonglong2 v0{0, 0}, v1{0, 0};
                if (comp < 3) {
                    v0 = *reinterpret_cast<const ulonglong2*>(p + l);
                    v1 = *reinterpret_cast<const ulonglong2*>(p + l + 2);
                }
                tm_wait();
                tm_pin(y);
                v0.x = gl_add(v0.x, join_wide(y.l));
                v0.y = gl_add(v0.y, join_wide(y.l + 8));
                v1.x = gl_add(v1.x, join_wide(y.l + 16));
                v1.y = gl_add(v1.y, join_wide(y.l + 24));
                if (comp < 3 && ok) {
                    *reinterpret_cast<ulonglong2*>(p + l) = v0;
                    *reinterpret_cast<ulonglong2*>(p + l + 2) = v1;
                }
            }
        }
    }
    if (!ok && a.err) atomicOr(a.err, TX_ERR_TIMEOUT);
    tc_before();
    __syncthreads();
    if (warp == 0) {
        tc_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
    }
}

}  // namespace

int cov_gemm_prepare() {
    return cudaFuncSetAttribute(k_cov_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CG_SMEM) == cudaSuccess ? 0 : -1;
}

// Returns 1 (nothing launched) when the form does not apply: vectors below 2^14
// (whose rows would not fill a 128-row tile, and whose update takes 22 us either
// way), or no room for the operand images in a.big.
int launch_cov_gemm(const CovAccArgs& a, cudaStream_t st) {
    u32 lg = 0;
    while ((1ull << lg) < a.size) ++lg;
    if (lg < 14 || lg > 26 || a.size != 1ull << lg || !a.big || (reinterpret_cast<uintptr_t>(a.big) & 15)) return 1;
    const u32 words = 3 * a.n_ext + a.n_base, chunks = (words + 15) / 16;
    const u32 log_lo = std::min(lg / 2, 10u), log_hi = lg - log_lo;
    const u32 rows = 3u << log_hi, tiles = (rows + 127) / 128, cols = 1u << (log_lo - 5);
    const size_t bytesA = (size_t)tiles * chunks * BLK, bytesB = (size_t)cols * chunks * 2 * BLK;
    if (bytesA + bytesB > a.big_bytes || words == 0 || ((u64)chunks * 16 << std::max(log_lo, log_hi)) >> 30) return 1;
    CovGemmArgs g{};
    for (int c = 0; c < 3; ++c) {
        g.cov[c] = a.cov[c];
        if (reinterpret_cast<uintptr_t>(a.cov[c]) & 15) return 1;
    }
    g.log_lo = log_lo;
    g.log_hi = log_hi;
    g.rows = rows;
    g.chunks = chunks;
    unsigned char* A = static_cast<unsigned char*>(a.big);
    g.A = A;
    g.B = A + bytesA;
    g.err = a.err;
    const u64 entries = (u64)chunks * 16 * ((1u << log_lo) + (1u << log_hi));
    k_cov_gemm_tables<<<(unsigned)std::min<u64>((entries + 255) / 256, 8ull * device_sms()), 256, 0, st>>>(
        a.sc, a.n_ext, a.n_base, log_lo, log_hi, chunks, A, A + bytesA, a.ext2 != 0);
    k_cov_gemm<<<dim3(cols, (tiles + 1) / 2), 32 * (CG_EPI_WARPS + 2), CG_SMEM, st>>>(g);
    count_launches(2);
    return 0;
}

}  // namespace wg
