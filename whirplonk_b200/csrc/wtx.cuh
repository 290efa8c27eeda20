// wtx.cuh -- the Fiat-Shamir transcript run by one warp.
//
// The byte semantics of transcript.cuh (the reference ProverState over a
// SHAKE128 duplex sponge, transcript.hpp:80-139, 375-453, 595-662); the sponge
// lives in registers of one warp: lane l < 25
// holds lane l of the hasher and of the XOF reader, Keccak-f[1600] runs with
// one state word per lane (theta / rho-pi / chi data exchange by shuffles), and
// aligned absorbs and squeezes move whole 8-byte words.  The bookkeeping values
// (positions, stream lengths) are warp-uniform; stream bytes are written by
// lane 0.
//
// Every function is warp-collective: all 32 lanes of the warp call it with the
// same arguments.  A kernel loads the state with wtx_load, runs its steps and
// writes it back with wtx_store.
#pragma once
#include "state.cuh"
#include "transcript.cuh"

namespace wg {

struct WarpTx {
    u64 h, r;  // this lane's hasher / reader word (lanes 0..24)
    unsigned hpos, rpos, has_reader, err, deg;
    u64 narg_len, hints_len, narg_cap, hints_cap;
    u8* narg;
    u8* hints;
};

__device__ __forceinline__ unsigned wtx_lane() { return threadIdx.x & 31; }

// The rho offsets of ten consecutive lanes from l0, six bits each.
__host__ __device__ constexpr u64 keccak_rho_pack(int l0) {
    u64 v = 0;
    for (int i = 0; i < 10 && l0 + i < 25; ++i) v |= (u64)keccak_rho((l0 + i) % 5, (l0 + i) / 5) << (6 * i);
    return v;
}

// Keccak-f[1600] with state word l in lane l.  Lane (x, y) = x + 5 y.  Each lane
// rotates its own word (rho), then fetches the three pi-permuted words chi needs
// -- B[X][Y], B[X+1][Y], B[X+2][Y] -- straight from their source lanes: three
// shuffle stages per round (theta's column sums, theta's D, pi + chi).  pi moves
// A[x][y] to (y, 2x + 3y), so lane (X, Y) receives from ((X + 3Y) mod 5, X).
// Nothing reads lanes 25..31.
//
// Bound by the 18 shuffles a round (~9 cycles each from one warp).  The words are
// kept as halves, so that a rotation is two selects and two funnel shifts (64-bit
// shifts: +4 %), and the lane's sources are a few instructions (25 compares for
// the offset and a dozen remainders: +~0.3 us a call).
static __device__ __noinline__ u64 keccak_f1600_warp(u64 a) {
    const unsigned l = wtx_lane();
    auto div5 = [](unsigned v) { return (v * 13) >> 6; };  // v < 32
    auto mod5 = [](unsigned v) { return v >= 5 ? v - 5 : v; };  // v < 10
    const unsigned y = div5(l), x = l - 5 * y;
    const unsigned v = x + 3 * y, s = v - 5 * div5(v);
    unsigned th[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) th[k] = x + 5 * mod5(y + 1 + k);
    const unsigned x1 = mod5(x + 1), cl = mod5(x + 4) + 5 * y, cr = x1 + 5 * y;
    const unsigned p0 = s + 5 * x, p1 = mod5(s + 1) + 5 * x1, p2 = mod5(s + 2) + 5 * mod5(x + 2);
    const unsigned g = l < 10 ? 0u : l < 20 ? 10u : 20u;
    const u64 pack = l < 10 ? keccak_rho_pack(0) : l < 20 ? keccak_rho_pack(10) : keccak_rho_pack(20);
    const unsigned rot = (unsigned)(pack >> (6 * ((l - g) % 10))) & 63;
    const bool swap = rot & 32;
    const unsigned rs = rot & 31, mask = l == 0 ? ~0u : 0u;
    unsigned lo = (unsigned)a, hi = (unsigned)(a >> 32);
#pragma unroll 1
    for (int round = 0; round < 24; ++round) {
        const u64 rc = KECCAK_RC[round];
        unsigned s0[4], s1[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            s0[k] = __shfl_sync(0xFFFFFFFFu, lo, th[k]);
            s1[k] = __shfl_sync(0xFFFFFFFFu, hi, th[k]);
        }
        const unsigned c0 = (lo ^ s0[0] ^ s0[1]) ^ s0[2] ^ s0[3], c1 = (hi ^ s1[0] ^ s1[1]) ^ s1[2] ^ s1[3];
        const unsigned e0 = __shfl_sync(0xFFFFFFFFu, c0, cr), e1 = __shfl_sync(0xFFFFFFFFu, c1, cr);
        const unsigned g0 = __shfl_sync(0xFFFFFFFFu, c0, cl), g1 = __shfl_sync(0xFFFFFFFFu, c1, cl);
        const unsigned t0 = lo ^ g0 ^ __funnelshift_l(e1, e0, 1), t1 = hi ^ g1 ^ __funnelshift_l(e0, e1, 1);
        const unsigned u0 = swap ? t1 : t0, u1 = swap ? t0 : t1;
        const unsigned r0 = __funnelshift_l(u1, u0, rs), r1 = __funnelshift_l(u0, u1, rs);
        const unsigned a0 = __shfl_sync(0xFFFFFFFFu, r0, p0), a1 = __shfl_sync(0xFFFFFFFFu, r1, p0);
        const unsigned b0 = __shfl_sync(0xFFFFFFFFu, r0, p1), b1 = __shfl_sync(0xFFFFFFFFu, r1, p1);
        const unsigned d0 = __shfl_sync(0xFFFFFFFFu, r0, p2), d1 = __shfl_sync(0xFFFFFFFFu, r1, p2);
        lo = (a0 ^ (~b0 & d0)) ^ ((unsigned)rc & mask);
        hi = (a1 ^ (~b1 & d1)) ^ ((unsigned)(rc >> 32) & mask);
    }
    return (u64)hi << 32 | lo;
}

__device__ __forceinline__ void wtx_load(WarpTx& t, const TxState* g) {
    const unsigned l = wtx_lane();
    t.h = l < 25 ? g->hasher[l] : 0;
    t.r = l < 25 ? g->reader[l] : 0;
    t.hpos = g->hpos;
    t.rpos = g->rpos;
    t.has_reader = g->has_reader;
    t.err = g->err;
    t.deg = g->deg;
    t.narg_len = g->narg_len;
    t.hints_len = g->hints_len;
    t.narg_cap = g->narg_cap;
    t.hints_cap = g->hints_cap;
    t.narg = g->narg;
    t.hints = g->hints;
}
__device__ __forceinline__ void wtx_store(const WarpTx& t, TxState* g) {
    const unsigned l = wtx_lane();
    if (l < 25) {
        g->hasher[l] = t.h;
        g->reader[l] = t.r;
    }
    if (l == 0) {
        g->hpos = t.hpos;
        g->rpos = t.rpos;
        g->has_reader = t.has_reader;
        g->err = t.err;
        g->deg = t.deg;
        g->narg_len = t.narg_len;
        g->hints_len = t.hints_len;
        g->narg_cap = t.narg_cap;
        g->hints_cap = t.hints_cap;
        g->narg = t.narg;
        g->hints = t.hints;
    }
    __syncwarp();
}

// absorb: continue the hasher; a pending reader is dropped.
__device__ __forceinline__ void wtx_absorb_byte(WarpTx& t, u8 v) {
    if (wtx_lane() == (t.hpos >> 3)) t.h ^= (u64)v << (8 * (t.hpos & 7));
    if (++t.hpos == TX_RATE) {
        t.h = keccak_f1600_warp(t.h);
        t.hpos = 0;
    }
}
// The first nw (<= N) words of w.  At a word boundary every word goes to its lane
// in one pass; word by word, each with its own test for a full block, took ~190
// cycles a word on B200.
template <int N>
__device__ __forceinline__ void wtx_absorb_words(WarpTx& t, const u64 (&w)[N], unsigned nw) {
    static_assert(8 * N <= TX_RATE, "at most one block boundary");
    constexpr unsigned RW = TX_RATE / 8;
    t.has_reader = 0;
    if ((t.hpos & 7) == 0) {
        const unsigned at = t.hpos >> 3, k = wtx_lane() - at;  // this lane takes word k of the block
        u64 v = 0, next = 0;
#pragma unroll
        for (unsigned i = 0; i < N; ++i)
            if (i < nw) {
                if (k == i) v = w[i];
                if (k + RW == i) next = w[i];
            }
        if (wtx_lane() < RW) t.h ^= v;
        t.hpos += 8 * nw;
        if (t.hpos >= TX_RATE) {
            t.h = keccak_f1600_warp(t.h) ^ next;
            t.hpos -= TX_RATE;
        }
        return;
    }
#pragma unroll 1
    for (unsigned i = 0; i < 8 * nw; ++i) {
        u64 v = 0;
#pragma unroll
        for (unsigned q = 0; q < N; ++q)
            if (q == i >> 3) v = w[q];
        wtx_absorb_byte(t, (u8)(v >> (8 * (i & 7))));
    }
}
// n bytes from memory, a lane the up to eight bytes of its word (byte by byte over
// the warp they took ~20 cycles each).
__device__ __forceinline__ void wtx_absorb_bytes(WarpTx& t, const u8* src, unsigned n) {
    t.has_reader = 0;
    while (n > 0) {
        const unsigned take = min(n, TX_RATE - t.hpos);
        u64 v = 0;
#pragma unroll
        for (unsigned b = 0; b < 8; ++b) {
            const unsigned i = 8 * wtx_lane() + b - t.hpos;
            if (i < take) v |= (u64)src[i] << (8 * b);
        }
        t.h ^= v;
        t.hpos += take;
        src += take;
        n -= take;
        if (t.hpos == TX_RATE) {
            t.h = keccak_f1600_warp(t.h);
            t.hpos = 0;
        }
    }
}

// The first squeeze after an absorb finalises a copy of the hasher.
__device__ __forceinline__ void wtx_reader(WarpTx& t) {
    if (t.has_reader) return;
    const unsigned l = wtx_lane();
    u64 r = t.h;
    if (l == (t.hpos >> 3)) r ^= (u64)0x1F << (8 * (t.hpos & 7));
    if (l == (TX_RATE - 1) >> 3) r ^= (u64)0x80 << (8 * ((TX_RATE - 1) & 7));
    t.r = keccak_f1600_warp(r);
    t.rpos = 0;
    t.has_reader = 1;
}
// n squeezed bytes into dst (shared or global memory), written by the warp.
__device__ __forceinline__ void wtx_squeeze_bytes(WarpTx& t, u8* dst, unsigned n) {
    if (n == 0) return;
    wtx_reader(t);
    const unsigned l = wtx_lane();
    unsigned done = 0;
    while (done < n) {
        if (t.rpos == TX_RATE) {
            t.r = keccak_f1600_warp(t.r);
            t.rpos = 0;
        }
        const unsigned take = min(n - done, TX_RATE - t.rpos);
        // every lane runs the same iterations so that all shuffles are full-warp
        for (unsigned k0 = 0; k0 < take; k0 += 32) {
            const unsigned k = k0 + l;
            const unsigned pos = t.rpos + (k < take ? k : take - 1);
            const u64 w = __shfl_sync(0xFFFFFFFFu, t.r, pos >> 3);
            if (k < take) dst[done + k] = (u8)(w >> (8 * (pos & 7)));
        }
        done += take;
        t.rpos += take;
    }
    __syncwarp();
}

// The first nw (<= N) words of w to the proof string, lane i word i.
template <int N>
__device__ __forceinline__ void wtx_narg_words(WarpTx& t, const u64 (&w)[N], unsigned nw) {
    if (t.narg_len + 8 * nw > t.narg_cap) {
        t.err |= TX_ERR_NARG_OVERFLOW;
        return;
    }
    const unsigned l = wtx_lane();
    u64 v = 0;
#pragma unroll
    for (unsigned i = 0; i < N; ++i)
        if (l == i) v = w[i];
    u8* dst = t.narg + t.narg_len + 8 * l;
    if (l < nw) {
        if ((reinterpret_cast<u64>(dst) & 7) == 0) {
            *reinterpret_cast<u64*>(dst) = v;
        } else {
#pragma unroll 1
            for (int b = 0; b < 8; ++b) dst[b] = (u8)(v >> (8 * b));
        }
    }
    t.narg_len += 8 * nw;
}
template <int N>
__device__ __forceinline__ void wtx_message_words(WarpTx& t, const u64 (&w)[N], unsigned nw = N) {
    wtx_absorb_words(t, w, nw);
    wtx_narg_words(t, w, nw);
}
__device__ __forceinline__ void wtx_message_u64(WarpTx& t, u64 v) {
    const u64 w[1] = {v};
    wtx_message_words(t, w);
}

// ncomp (<= 3) consecutive base-field challenges, challenge c in component c:
// 40 squeezed bytes each as a LE integer mod p (five words folded from the top).
// Lane c gathers the six state words that hold challenge c at any alignment -- the
// index bytes of an opening leave the reader between words -- from this block and,
// past its end, the next.  (Byte by byte an unaligned Ext3 challenge took ~12 k
// cycles on B200, this ~1 k.)
__device__ __forceinline__ E3 wtx_challenges(WarpTx& t, u32 ncomp) {
    constexpr u32 RW = TX_RATE / 8;
    wtx_reader(t);
    const unsigned l = wtx_lane();
    const u32 end = t.rpos + 40 * ncomp, sh = 8 * (t.rpos & 7);
    const u32 src = (t.rpos >> 3) + (l < ncomp ? 5 * l : 0);
    u64 w[6];
#pragma unroll
    for (u32 q = 0; q < 6; ++q) w[q] = __shfl_sync(0xFFFFFFFFu, t.r, src + q);
    if (end > TX_RATE) {
        t.r = keccak_f1600_warp(t.r);
#pragma unroll
        for (u32 q = 0; q < 6; ++q) {
            const u64 v = __shfl_sync(0xFFFFFFFFu, t.r, src + q - RW);
            if (src + q >= RW) w[q] = v;
        }
    }
    t.rpos = end > TX_RATE ? end - TX_RATE : end;
    u64 s = 0;
#pragma unroll
    for (int q = 4; q >= 0; --q) s = gl_reduce(sh ? (w[q] >> sh) | (w[q + 1] << (64 - sh)) : w[q], s);
    const u64 c0 = __shfl_sync(0xFFFFFFFFu, s, 0);
    const u64 c1 = __shfl_sync(0xFFFFFFFFu, s, 1);
    const u64 c2 = __shfl_sync(0xFFFFFFFFu, s, 2);
    return E3{c0, ncomp > 1 ? c1 : 0, ncomp > 2 ? c2 : 0};
}
__device__ __forceinline__ u64 wtx_challenge_base(WarpTx& t) { return wtx_challenges(t, 1).c0; }

// Elements of the protocol's target field.  With the base field as target
// (Identity<Goldilocks>) its elements are carried as Ext3 values (x, 0, 0) --
// a subfield, so every kernel's arithmetic is unchanged -- and cross the
// transcript as one 8-byte word / one 40-byte challenge; GoldilocksExt2
// elements are carried as (c0, c1, 0) (products folded by e2_fold) and cross
// it as two words / two 40-byte chunks (transcript.hpp:375-453).
__device__ __forceinline__ E3 wtx_challenge_t(WarpTx& t) {
    return wtx_challenges(t, t.deg == 1 ? 1u : (t.deg == 2 ? 2u : 3u));
}
__device__ __forceinline__ void wtx_check_t(WarpTx& t, const E3& v) {  // caller input outside the target field
    if ((t.deg == 1 && v.c1) || (t.deg <= 2 && v.c2)) t.err |= TX_ERR_FIELD;
}
__device__ __forceinline__ void wtx_narg_t(WarpTx& t, const E3& v) {
    const u64 w[3] = {v.c0, v.c1, v.c2};
    wtx_narg_words(t, w, t.deg);
}
__device__ __forceinline__ void wtx_message_t(WarpTx& t, const E3& v) {
    wtx_check_t(t, v);
    const u64 w[3] = {v.c0, v.c1, v.c2};
    wtx_message_words(t, w, t.deg);
}
// Two consecutive messages, absorbed in one pass and not yet in the proof string:
// the caller appends them (wtx_narg_t) once the challenge has been handed on.
__device__ __forceinline__ void wtx_absorb2_t(WarpTx& t, const E3& x, const E3& y) {
    wtx_check_t(t, x);
    wtx_check_t(t, y);
    const bool d1 = t.deg == 1, d2 = t.deg == 2;
    const u64 w[6] = {x.c0, d1 ? y.c0 : x.c1, d2 ? y.c0 : x.c2, d2 ? y.c1 : y.c0, y.c1, y.c2};
    wtx_absorb_words(t, w, 2 * t.deg);
}

// A PoW's challenge (proof_of_work.hpp), and the search's state reset.
__device__ __forceinline__ void wtx_pow_challenge(WarpTx& t, ProofScalars* sc) {
    wtx_squeeze_bytes(t, sc->pow_ch, 32);
    if (wtx_lane() == 0) {
        sc->pow_best = ~0ull;
        sc->pow_next = 0;
    }
}

// geometric_challenge (geometric_challenge.hpp:39-44): [] / [1] / squeeze x ->
// [1, x, x^2, ...]; the powers are formed 32 at a time (lane k: x^(32 j + k)).
__device__ __forceinline__ void wtx_geometric(WarpTx& t, E3* out, int count) {
    if (count <= 0) return;
    const unsigned l = wtx_lane();
    if (count == 1) {
        if (l == 0) out[0] = e3_one();
        __syncwarp();
        return;
    }
    const E3 x = wtx_challenge_t(t);
    // lane k: x^k by an in-warp prefix product (Hillis-Steele on multipliers;
    // rolled: one copy of the product's code to fetch)
    E3 p = l == 0 ? e3_one() : x;
#pragma unroll 1
    for (int o = 1; o < 32; o <<= 1) {
        const E3 q{__shfl_up_sync(0xFFFFFFFFu, p.c0, o), __shfl_up_sync(0xFFFFFFFFu, p.c1, o),
                   __shfl_up_sync(0xFFFFFFFFu, p.c2, o)};
        if (l >= (unsigned)o) p = ef_mul(p, q, t.deg == 2);
    }
    // x^32 = (x^31) * x
    E3 x31{__shfl_sync(0xFFFFFFFFu, p.c0, 31), __shfl_sync(0xFFFFFFFFu, p.c1, 31), __shfl_sync(0xFFFFFFFFu, p.c2, 31)};
    const E3 x32 = ef_mul(x31, x, t.deg == 2);
    for (int base = 0; base < count; base += 32) {
        if (base + (int)l < count) out[base + l] = p;
        p = ef_mul(p, x32, t.deg == 2);
    }
    __syncwarp();
}

// Warp-wide field sum (exact; association order free).
__device__ __forceinline__ E3 wtx_sum(E3 v) { return e3_warp_sum(v); }

// Vector RLC, constraint RLC and "the sum" (whir_prover.hpp:122-197):
//   vrlc = geometric_challenge(V), crlc = geometric_challenge(F + O),
//   sum  = sum_f crlc_f sum_v vrlc_v eval_(f,v) + sum_i crlc_(F+i) sum_v vrlc_v ood_(i,v)
// over the O = nwit * ood initial OOD points, whose coordinates are also laid
// out contiguously for the covector.  One warp.
__device__ __forceinline__ void wtx_constraint_rlc(TxState* tx, ProofScalars* sc, int n_forms, int nwit, int ood, int nvec) {
    const int l = wtx_lane();
    const int n_ood = nwit * ood;
    for (int i = l; i < n_ood; i += 32) sc->init_ood_pts[i] = sc->ood_pts[i / ood][i % ood];
    const int count = n_forms + n_ood;
    WarpTx t;
    wtx_load(t, tx);
    wtx_geometric(t, sc->vrlc, nvec);
    wtx_geometric(t, sc->crlc, count);
    wtx_store(t, tx);
    E3 v = e3_zero();
    for (int r = l; r < count; r += 32) {
        const E3* vals = r < n_forms ? &sc->forms_eval[r * nvec] : &sc->init_ood_mat[(r - n_forms) * nvec];
        E3 row = e3_zero();
        for (int k = 0; k < nvec; ++k) row = e3_add(row, ef_mul(sc->vrlc[k], vals[k], t.deg == 2));
        v = e3_add(v, ef_mul(sc->crlc[r], row, t.deg == 2));
    }
    v = wtx_sum(v);
    if (l == 0) sc->sum = v;
}

}  // namespace wg
