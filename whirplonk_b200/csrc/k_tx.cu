// k_tx.cu -- the sequential Fiat-Shamir steps of the prover, executed on the
// device: transcript start, constraint/STIR combination challenges, proof of
// work grinding, in-domain openings (indices, row hints, Merkle paths) and
// the final-vector message.  Protocol order and byte layout follow
// cpp/include/whir/protocols/whir/whir_prover.hpp:56-407.
#include <algorithm>

#include "launch.h"
#include "blake3.cuh"
#include "sha256.cuh"
#include "state.cuh"
#include "wtx.cuh"

namespace wg {

// ---------------------------------------------------------------------------
// Transcript start: ProverState::from_ds (transcript.hpp:605-610) absorbs
// protocol_id || session_id || instance bytes.
// ---------------------------------------------------------------------------
// One warp.
__global__ void k_tx_init(TxState* tx, const unsigned char* ds, u32 ds_len, unsigned char* narg, u64 narg_cap,
                          unsigned char* hints, u64 hints_cap, ProofScalars* sc, unsigned deg) {
    if (threadIdx.x >= 32) return;
    WarpTx t;
    t.h = t.r = 0;
    t.hpos = t.rpos = t.has_reader = t.err = 0;
    t.deg = deg;
    t.narg_len = t.hints_len = 0;
    t.narg_cap = narg_cap;
    t.hints_cap = hints_cap;
    t.narg = narg;
    t.hints = hints;
    wtx_absorb_bytes(t, ds, ds_len);
    wtx_store(t, tx);
    for (int i = threadIdx.x; i < 64; i += 32) sc->counters[i] = 0;
}

int launch_tx_init(TxState* tx, const unsigned char* ds, u32 ds_len, unsigned char* narg, u64 narg_cap,
                   unsigned char* hints, u64 hints_cap, ProofScalars* sc, unsigned deg, cudaStream_t st) {
    if (deg < 1 || deg > 3) return -1;
    k_tx_init<<<1, 32, 0, st>>>(tx, ds, ds_len, narg, narg_cap, hints, hints_cap, sc, deg);
    count_launches(1);
    return 0;
}

__global__ void k_constraint_rlc(TxState* tx, ProofScalars* sc, int n_forms, int nwit, int ood, int nvec) {
    if (threadIdx.x < 32) wtx_constraint_rlc(tx, sc, n_forms, nwit, ood, nvec);
}

int launch_constraint_rlc(TxState* tx, ProofScalars* sc, int n_forms, int nwit, int ood, int nvec, cudaStream_t st) {
    if (n_forms > MAX_FORMS || ood > MAX_OOD || nwit < 1 || nwit > MAX_WITNESSES || nvec < 1 || nvec > MAX_VECTORS)
        return -1;
    k_constraint_rlc<<<1, 32, 0, st>>>(tx, sc, n_forms, nwit, ood, nvec);
    count_launches(1);
    return 0;
}

// ---------------------------------------------------------------------------
// Proof of work (proof_of_work.hpp:95-193, 236-257): the smallest nonce n >= 0
// with LE_u64(BLAKE3(challenge || n_le || 0^24)[0..8]) <= threshold.
//
// One launch: CTAs claim chunks of POW_CHUNK consecutive nonces in increasing
// order from a counter (atomicAdd), scan a claimed chunk completely and claim
// the next one while the previous hit published in pow_best (atomicMin) is not
// below the chunk.  Every chunk that starts at or below the final minimum is
// therefore claimed and fully scanned, so the minimum is exact -- the
// reference's answer, whatever the scheduling -- and the work past it is at
// most one chunk per CTA.  The search stops at 64x the expected length
// 2^64 / threshold (miss probability e^-64), capped at POW_NONCE_LIMIT; running
// out sets TX_ERR_POW_EXHAUSTED.
// ---------------------------------------------------------------------------
constexpr u64 POW_NONCE_LIMIT = 1ull << 36;
constexpr unsigned POW_THREADS = 256, POW_CTAS_PER_SM = 2, POW_CTAS_LONG = 3, POW_CHUNK = 2 * POW_THREADS;

// One warp.  Also resets the search state.
__global__ void k_pow_challenge(TxState* tx, ProofScalars* sc) {
    if (threadIdx.x >= 32) return;
    WarpTx t;
    wtx_load(t, tx);
    wtx_pow_challenge(t, sc);
    wtx_store(t, tx);
}

// H: 0 = BLAKE3, 1 = SHA-256 (the PoW engine follows the hash_id, whir.hpp:134-140).
// Most of a nonce's message words are zero, which leaves BLAKE3's additions fewer than
// its rotations: additions on the FMA pipe are slower here (34.1 G nonces/s on B200
// against 36.6, two CTAs an SM), unlike in the trees.  SHA-256: 9.74 against 9.40.
template <int H>
__global__ void __launch_bounds__(POW_THREADS) k_pow_search(ProofScalars* sc, u64 threshold, u64 limit) {
    __shared__ unsigned ch[8];
    __shared__ u64 claim[2];
    __shared__ int stop;
    unsigned long long* next = reinterpret_cast<unsigned long long*>(&sc->pow_next);
    if (threadIdx.x < 8) {
        const unsigned char* c = sc->pow_ch + 4 * threadIdx.x;
        ch[threadIdx.x] = (unsigned)c[0] | ((unsigned)c[1] << 8) | ((unsigned)c[2] << 16) | ((unsigned)c[3] << 24);
    }
    if (threadIdx.x == 0) claim[0] = atomicAdd(next, (unsigned long long)POW_CHUNK);
    __syncthreads();
    unsigned m[16];
#pragma unroll
    for (int k = 0; k < 8; ++k) m[k] = ch[k];
#pragma unroll
    for (int k = 10; k < 16; ++k) m[k] = 0;
    for (unsigned it = 0;; ++it) {
        const u64 base = claim[it & 1];
        if (threadIdx.x == 0) {
            stop = base >= limit || base > __ldcg(&sc->pow_best);
            // claim the next chunk now, so the counter's latency overlaps the hashing
            if (!stop) claim[(it + 1) & 1] = atomicAdd(next, (unsigned long long)POW_CHUNK);
        }
        __syncthreads();
        if (stop) break;
#pragma unroll
        for (unsigned k = 0; k < POW_CHUNK / POW_THREADS; ++k) {
            const u64 n = base + k * POW_THREADS + threadIdx.x;
            if (n >= limit) break;
            m[8] = (unsigned)n;
            m[9] = (unsigned)(n >> 32);
            unsigned h[8];
            if (H == 1) sha256_hash64(m, h);
            else b3_hash64<false>(m, h);
            const u64 v = (u64)h[0] | ((u64)h[1] << 32);  // first 8 digest bytes, LE
            if (v <= threshold) atomicMin(reinterpret_cast<unsigned long long*>(&sc->pow_best), (unsigned long long)n);
        }
        __syncthreads();
    }
}

// The search for one PoW (challenge already squeezed, pow_best / pow_next reset).
int launch_pow_grind_only(ProofScalars* sc, u64 threshold, int hash, cudaStream_t st) {
    const double expect = threshold == 0 ? 1.8446744073709552e19 : 18446744073709551616.0 / (double)threshold;
    const u64 limit = expect * 64.0 >= (double)POW_NONCE_LIMIT ? POW_NONCE_LIMIT : (u64)(expect * 64.0) + 1;
    // Every CTA finishes the chunk it holds when the minimum turns up, so the
    // work past the answer is about one chunk per CTA: a search expected to be
    // short gets one CTA per SM (the latency of a proof alone stays that of a
    // full grid), a long one up to POW_CTAS_PER_SM per SM.  The answer does not
    // depend on the grid.
    const double want = expect / (4.0 * POW_CHUNK);
    // (From 2^24 expected nonces up the third CTA's overshoot is below 2 %: 38.4 against
    // 36.6 G nonces/s.)
    const unsigned sms = device_sms(), cap = (expect >= 0x1p24 ? POW_CTAS_LONG : POW_CTAS_PER_SM) * sms;
    const unsigned grid = want >= (double)cap ? cap : (want <= (double)sms ? sms : (unsigned)want);
    if (hash == 1) k_pow_search<1><<<grid, POW_THREADS, 0, st>>>(sc, threshold, limit);
    else k_pow_search<0><<<grid, POW_THREADS, 0, st>>>(sc, threshold, limit);
    count_launches(1);
    return 0;
}

__global__ void k_pow_finish(TxState* tx, ProofScalars* sc, int slot) {
    if (threadIdx.x >= 32) return;
    const u64 n = sc->pow_best;
    WarpTx t;
    wtx_load(t, tx);
    if (n == ~0ull) t.err |= TX_ERR_POW_EXHAUSTED;
    if (threadIdx.x == 0 && slot >= 0 && slot < MAX_COMMITS + 4) sc->pow_nonces[slot] = n;
    wtx_message_u64(t, n);
    wtx_store(t, tx);
}

int launch_pow_search(TxState* tx, ProofScalars* sc, u64 threshold, int hash, bool drawn, cudaStream_t st) {
    if (threshold == ~0ull) return 0;  // zero difficulty: nothing sent (proof_of_work.hpp:241)
    if (!drawn) {
        k_pow_challenge<<<1, 32, 0, st>>>(tx, sc);
        count_launches(1);
    }
    return launch_pow_grind_only(sc, threshold, hash, st);
}
int launch_pow(TxState* tx, ProofScalars* sc, u64 threshold, int slot, int hash, cudaStream_t st) {
    if (threshold == ~0ull) return 0;
    launch_pow_search(tx, sc, threshold, hash, false, st);
    k_pow_finish<<<1, 32, 0, st>>>(tx, sc, slot);
    count_launches(1);
    return 0;
}

// Final vector: prover_message of every coefficient (whir_prover.hpp:360-362).
// One warp; pow_sc: the challenge of the PoW that follows, too.
__global__ void k_send_vector(TxState* tx, const u64* c0, const u64* c1, const u64* c2, u64 size, ProofScalars* pow_sc) {
    if (threadIdx.x >= 32) return;
    WarpTx t;
    wtx_load(t, tx);
    for (u64 i = 0; i < size; ++i) wtx_message_t(t, E3{c0[i], c1[i], c2[i]});
    if (pow_sc) wtx_pow_challenge(t, pow_sc);
    wtx_store(t, tx);
}

int launch_send_vector(TxState* tx, const u64* c0, const u64* c1, const u64* c2, u64 size, ProofScalars* pow_sc,
                       cudaStream_t st) {
    k_send_vector<<<1, 32, 0, st>>>(tx, c0, c1, c2, size, pow_sc);
    count_launches(1);
    return 0;
}

// `count` Ext3 challenges in a row into sc->sc_r[slot ..] -- the folding
// randomness of a proof without constraints (whir_prover.hpp:211-218,
// verifier_message_vec).  One warp.
__global__ void k_squeeze_e3(TxState* tx, ProofScalars* sc, int slot, int count) {
    if (threadIdx.x >= 32) return;
    WarpTx t;
    wtx_load(t, tx);
    for (int k = 0; k < count; ++k) {
        const E3 r = wtx_challenge_t(t);
        if (threadIdx.x == 0) sc->sc_r[slot + k] = r;
    }
    wtx_store(t, tx);
}

int launch_squeeze_challenges(TxState* tx, ProofScalars* sc, int slot, int count, cudaStream_t st) {
    if (count <= 0) return 0;
    if (slot < 0 || slot + count > MAX_SC_ROUNDS) return -1;
    k_squeeze_e3<<<1, 32, 0, st>>>(tx, sc, slot, count);
    count_launches(1);
    return 0;
}

// ---------------------------------------------------------------------------
// Opening (irs_commit.hpp:600-713, challenge_indices.hpp:56-119,
// merkle_tree.hpp:165-211) of nwit commitments at the same rows:
//   0. (after a PoW search) the nonce message (proof_of_work.hpp);
//   1. squeeze q * ceil(log2(N)/8) bytes, index = big-endian bytes mod N;
//   2. per commitment: hint u64 (q * depth), the q rows in index order
//      (duplicates kept), then its Merkle hints -- sorted, deduplicated
//      indices climbed level by level, a node's sibling is emitted unless the
//      sibling is itself in the set.  Every commitment has the same tree shape
//      and indices, so its hint block has the same length;
//   3. (STIR) point gen^idx and value <rows, vector_rlc (x) eq_weights(last
//      folding randomness)> over the rows of all commitments side by side
//      (whir_prover.hpp:283-310);
//   4. (STIR) the combination over the new commitment's OOD points/values and
//      these: RLC = geometric_challenge(O + q), sum += <rlc, values>
//      (whir_prover.hpp:310-336).
//
// A chain of dependent loads and transcript steps, so latency is all that
// counts.  Warp 0 of a CTA runs the transcript -- nonce, index bytes, then the
// RLC challenge and its powers, which wait for no value -- while the other
// warps sort the indices and gather rows, values and hashes.  Up to OPEN_CTAS
// CTAs do the transcript and the sort each for itself (the same bytes; no CTA
// waits for another) and share the gathering; the last one to finish (a
// self-resetting ticket) sums the combination and stores the transcript.
// Against one CTA of 1024 threads between a nonce launch and a combination
// launch (B200, a whole proof): n = 16 rate 1/4 823 -> 766 us, n = 18 rate 1/2
// 1007 -> 935 us.  The same split with the powers after the values gained 20 us
// less.
// ---------------------------------------------------------------------------
constexpr int OPEN_THREADS = 512, OPEN_WARPS = OPEN_THREADS / 32;
constexpr int OPEN_GATHER = OPEN_THREADS - 32;  // threads of the gathering warps
constexpr int OPEN_SORT = 256;                  // of these, threads that sort while the others take the rows' values
constexpr u32 OPEN_ROW_WARPS = (OPEN_GATHER - OPEN_SORT) / 32;
constexpr u32 OPEN_CTAS = 8, OPEN_MAX_LOGN = 26;

// Barriers of the gathering and of the sorting warps, and the latter counting `v`.
__device__ __forceinline__ void gather_sync() { asm volatile("bar.sync 1, %0;" ::"n"(OPEN_GATHER) : "memory"); }
__device__ __forceinline__ void sort_sync() { asm volatile("bar.sync 2, %0;" ::"n"(OPEN_SORT) : "memory"); }
__device__ __forceinline__ u32 sort_count(bool v) {
    u32 r;
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.popc.u32 %0, 2, %2, p;\n\t}"
                 : "=r"(r)
                 : "r"((u32)v), "n"(OPEN_SORT)
                 : "memory");
    return r;
}

__global__ void __launch_bounds__(OPEN_THREADS) k_open(OpenArgs a) {
    __shared__ u64 idx_s[MAX_QUERIES];
    __shared__ u64 cur[MAX_QUERIES];
    __shared__ unsigned char dup[MAX_QUERIES];
    __shared__ E3 eqw[MAX_DEPTH];
    __shared__ unsigned char idx_bytes[MAX_QUERIES * 4];
    __shared__ u32 cnt[OPEN_MAX_LOGN][MAX_QUERIES / 32];  // emitted siblings per level and chunk of 32 nodes, then their prefix
    __shared__ u32 lvl[OPEN_MAX_LOGN + 1];                // siblings of the levels below, and of all
    __shared__ E3 red[OPEN_WARPS];
    __shared__ u64 gpow[32];  // gen^(2^i)
    __shared__ u32 distinct;
    __shared__ bool last;
    const TxState* tx = a.tx;  // the hint stream (unchanged until the last CTA's store)
    ProofScalars* sc = a.sc;
    const u32 t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const u32 q = a.q;
    const u32 nbytes = (a.logN + 7) / 8;
    const u32 nwit = a.nwit;
    const bool x2 = tx->deg == 2;  // GoldilocksExt2 target field
    const u64 hint_base = tx->hints_len;
    const int count = a.ood_offset + (int)q;  // values of the STIR combination

    WarpTx wt;
    if (warp == 0) {
        wtx_load(wt, a.tx);
        if (a.pow_slot >= 0) {
            const u64 n = sc->pow_best;
            if (n == ~0ull) wt.err |= TX_ERR_POW_EXHAUSTED;
            if (blockIdx.x == 0 && lane == 0 && a.pow_slot < MAX_COMMITS + 4) sc->pow_nonces[a.pow_slot] = n;
            wtx_message_u64(wt, n);
        }
        if (a.N != 1) wtx_squeeze_bytes(wt, idx_bytes, q * nbytes);
    } else if (a.stir) {
        // eq weights of the last `fold` folding challenges (multilinear_point.hpp:40-62)
        for (u32 i = t - 32; i < (1u << a.fold); i += OPEN_GATHER) {
            E3 acc = e3_one();
            for (u32 k = 0; k < a.fold; ++k) {
                const E3 r = sc->sc_r[a.r_offset + k];
                const bool bit = (i >> (a.fold - 1 - k)) & 1;
                acc = ef_mul(acc, bit ? r : e3_sub(e3_one(), r), x2);
            }
            eqw[i] = acc;
        }
        if (t == OPEN_THREADS - 1) {
            u64 p = a.gen;
            for (u32 i = 0; i < a.logN; ++i, p = gl_mul(p, p)) gpow[i] = p;
        }
    }
    __syncthreads();
    u64 blk = 0;  // hint bytes of one commitment (gathering warps)
    bool fits = true;
    if (warp == 0) {
        // Every CTA writes the same powers to the same place.
        if (a.stir) wtx_geometric(wt, sc->stir_rlc, count);
    } else {
        const u32 g = t - 32;  // gathering thread
        const u32 ggw = blockIdx.x * (OPEN_WARPS - 1) + warp - 1, ggws = gridDim.x * (OPEN_WARPS - 1);
        for (u32 i = g; i < q; i += OPEN_GATHER) {
            u64 acc = 0;
            for (u32 k = 0; k < nbytes; ++k) acc = (acc << 8) | idx_bytes[i * nbytes + k];
            acc = a.N == 1 ? 0 : (acc & (a.N - 1));  // N is a power of two
            idx_s[i] = acc;
            if (blockIdx.x == 0) sc->indices[i] = acc;
        }
        gather_sync();

        u32 u = 0;  // distinct indices
        // Merkle levels.  Per level L the nodes are the distinct values x of
        // cur[j] >> L (cur is sorted, so equal values are adjacent); x emits its
        // sibling x ^ 1 unless the sibling is itself a node, i.e. the
        // neighbouring distinct value: an odd x decides at its first j, an even
        // x at its last.  Siblings are emitted level by level, increasing x
        // within a level.
        auto emits = [&](u32 j, u32 L) -> bool {
            if (j >= u) return false;
            const u64 x = cur[j] >> L;
            if (x & 1) {
                if (j == 0) return true;
                const u64 p = cur[j - 1] >> L;
                return p != x && p != x - 1;
            }
            if (j + 1 == u) return true;
            const u64 n = cur[j + 1] >> L;
            return n != x && n != x + 1;
        };
        auto exclusive = [&](u32 v, u32& total) {
            u32 incl = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const u32 w = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                if (lane >= (u32)o) incl += w;
            }
            total = __shfl_sync(0xFFFFFFFFu, incl, 31);
            return incl - v;
        };
        if (warp <= OPEN_SORT / 32) {
            // Sort + dedup: a value goes to slot #{distinct values below it}.  Two
            // lanes share an index's comparisons.
            for (u32 i0 = 0; i0 < q; i0 += OPEN_SORT / 2) {
                const u32 i = i0 + (g >> 1);
                const u64 v = i < q ? idx_s[i] : 0;
                bool d = false;
                for (u32 j = g & 1; j < i && i < q; j += 2) d |= idx_s[j] == v;
                d |= __shfl_xor_sync(0xFFFFFFFFu, (int)d, 1);
                if (i < q) dup[i] = d;
                u += sort_count(i < q && !d && (g & 1) == 0);
            }
            for (u32 i0 = 0; i0 < q; i0 += OPEN_SORT / 2) {
                const u32 i = i0 + (g >> 1);
                const u64 v = i < q ? idx_s[i] : 0;
                u32 lt = 0;
                for (u32 j = g & 1; j < q; j += 2) lt += idx_s[j] < v && !dup[j];
                lt += __shfl_xor_sync(0xFFFFFFFFu, lt, 1);
                if (i < q && !dup[i] && (g & 1) == 0) cur[lt] = v;
            }
            sort_sync();

            const u32 chunks = (u + 31) / 32;
            for (u32 it = warp - 1; it < a.logN * chunks; it += OPEN_SORT / 32) {
                const u32 L = it / chunks, c = it % chunks;
                const u32 m = __popc(__ballot_sync(0xFFFFFFFFu, emits(c * 32 + lane, L)));
                if (lane == 0) cnt[L][c] = m;
            }
            sort_sync();
            for (u32 L = warp - 1; L < a.logN; L += OPEN_SORT / 32) {
                u32 total;
                const u32 e = exclusive(lane < chunks ? cnt[L][lane] : 0, total);
                if (lane < chunks) cnt[L][lane] = e;
                if (lane == 0) lvl[L] = total;
            }
            sort_sync();
            if (warp == 1) {
                u32 total;
                const u32 e = exclusive(lane < a.logN ? lvl[lane] : 0, total);
                if (lane <= a.logN) lvl[lane] = e;
            }
            if (g == 0) distinct = u;
        } else if (a.stir) {
            // 3. STIR point and value of each opened row: a warp per row, its lanes
            //    over the row's elements (all commitments side by side), a warp sum.
            const u32 dmask = (1u << a.fold) - 1;
            const u32 elems = nwit * a.depth;
            const u32 rows = gridDim.x * OPEN_ROW_WARPS;
            for (u32 i = blockIdx.x * OPEN_ROW_WARPS + warp - 1 - OPEN_SORT / 32; i < q; i += rows) {
                const u64 id = codeword_row(idx_s[i], a.logN, a.perm_log_e);  // natural row = exponent of its point
                u64 pt = lane < a.logN && ((id >> lane) & 1) ? gpow[lane] : 1;  // gen^id, a lane a bit
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) pt = gl_mul(pt, __shfl_xor_sync(0xFFFFFFFFu, pt, o));
                E3 val = e3_zero();
                for (u32 k = lane; k < elems; k += 32) {
                    const u32 w = k / a.depth, el = k - w * a.depth;
                    const u64* planes = a.planes + w * a.planes_stride;
                    E3 term;
                    if (a.ncomp == 1) {
                        term = e3_mul_base(eqw[el & dmask], planes[(u64)el * a.N + id]);
                    } else if (a.ncomp == 2) {  // Ext2 rows: planes c0, c1
                        term = ef_mul(E3{planes[(u64)el * a.N + id], planes[((u64)a.depth + el) * a.N + id], 0},
                                      eqw[el & dmask], true);
                    } else {
                        term = e3_mul(E3{planes[(u64)el * a.N + id], planes[((u64)a.depth + el) * a.N + id],
                                         planes[((u64)2 * a.depth + el) * a.N + id]},
                                      eqw[el & dmask]);
                    }
                    if (a.use_vrlc) term = ef_mul(term, sc->vrlc[w * (a.depth >> a.fold) + (el >> a.fold)], x2);
                    val = e3_add(val, term);
                }
                val = e3_warp_sum(val);
                if (lane == 0) {
                    sc->stir_pts[a.ood_offset + i] = e3_base(pt);
                    sc->stir_vals[a.ood_offset + i] = val;
                }
            }
        }
        gather_sync();
        u = distinct;
        const u32 nchunk = (u + 31) / 32;
        const u64 merkle_bytes = 32ull * lvl[a.logN];
        const u64 esz = 8ull * a.ncomp;
        const u64 row_bytes = esz * a.depth;
        const u64 row_hint = 8 + row_bytes * q;
        blk = row_hint + merkle_bytes;
        fits = hint_base + blk * nwit <= tx->hints_cap;

        // 2a. row hints.  Every hint word sits at a multiple of 8 bytes from the
        // commitment's hint block, so when the block starts 8-byte aligned (the
        // hints stream holds whole words) a word is one 8-byte store.
        const bool hints_al8 = (reinterpret_cast<uintptr_t>(tx->hints + hint_base) & 7) == 0;
        if (fits) {
            const u32 rw = a.depth * a.ncomp;  // words per row (<= MAX_DEPTH * 3)
            const u32 nwords = q * rw;
            for (u32 w = 0; w < nwit; ++w) {
                unsigned char* hb = tx->hints + hint_base + w * blk;
                const u64* planes = a.planes + w * a.planes_stride;
                if (g == 0 && blockIdx.x == 0) {
                    const u64 len = (u64)q * a.depth;
                    for (int k = 0; k < 8; ++k) hb[k] = (unsigned char)(len >> (8 * k));
                }
                for (u32 x = blockIdx.x * OPEN_GATHER + g; x < nwords; x += gridDim.x * OPEN_GATHER) {
                    const u32 qi = x / rw, rem = x - qi * rw;
                    const u32 el = rem / a.ncomp, c = rem - el * a.ncomp;
                    const u64 v = planes[((u64)c * a.depth + el) * a.N + codeword_row(idx_s[qi], a.logN, a.perm_log_e)];
                    unsigned char* dst = hb + 8 + qi * row_bytes + (u64)el * esz + 8ull * c;
                    if (hints_al8) {
                        *reinterpret_cast<u64*>(dst) = v;
                    } else {
#pragma unroll 1
                        for (int k = 0; k < 8; ++k) dst[k] = (unsigned char)(v >> (8 * k));
                    }
                }
            }
            // 2b. Merkle hints of every commitment: a warp per level and chunk.
            for (u32 it = ggw; it < a.logN * nchunk; it += ggws) {
                const u32 L = it / nchunk, c = it % nchunk;
                const u32 j = c * 32 + lane;
                const bool e = emits(j, L);
                const unsigned m = __ballot_sync(0xFFFFFFFFu, e);
                if (!e) continue;
                const u64 level_off = (2ull << a.logN) - (2ull << (a.logN - L));
                const u64 x = cur[j] >> L;
                const u64 rel = row_hint + 32ull * (lvl[L] + cnt[L][c] + __popc(m & ((1u << lane) - 1)));
                for (u32 w = 0; w < nwit; ++w) {
                    const u32* nodes = a.nodes + w * a.nodes_stride;
                    const uint4* src = reinterpret_cast<const uint4*>(nodes + (level_off + (x ^ 1)) * 8);
                    const uint4 h0 = src[0], h1 = src[1];
                    unsigned char* dst = tx->hints + hint_base + w * blk + rel;
                    if (hints_al8) {
                        u64* d8 = reinterpret_cast<u64*>(dst);
                        d8[0] = (u64)h0.x | ((u64)h0.y << 32);
                        d8[1] = (u64)h0.z | ((u64)h0.w << 32);
                        d8[2] = (u64)h1.x | ((u64)h1.y << 32);
                        d8[3] = (u64)h1.z | ((u64)h1.w << 32);
                    } else {
                        const unsigned w8[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
#pragma unroll 1
                        for (int k = 0; k < 32; ++k) dst[k] = (unsigned char)(w8[k >> 2] >> (8 * (k & 3)));
                    }
                }
            }
        }
    }

    // The last CTA: every CTA has read the transcript and written its values.
    __threadfence();
    __syncthreads();
    if (t == 32) {
        last = atomicAdd(&sc->counters[CTR_OPEN], 1u) == gridDim.x - 1;
        cur[0] = blk;  // to warp 0
        cur[1] = fits;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    if (a.stir) {
        if (t < (u32)a.ood_offset) {
            sc->stir_pts[t] = sc->ood_pts[a.rlc_commit][t];
            sc->stir_vals[t] = sc->ood_vals[a.rlc_commit][t];
        }
        E3 acc = e3_zero();
        for (int j = t; j < count; j += OPEN_THREADS) {
            const E3* v = j < a.ood_offset ? &sc->ood_vals[a.rlc_commit][j] : &sc->stir_vals[j];
            const E3* r = &sc->stir_rlc[j];
            acc = e3_add(acc, ef_mul(E3{__ldcg(&r->c0), __ldcg(&r->c1), __ldcg(&r->c2)},
                                     E3{__ldcg(&v->c0), __ldcg(&v->c1), __ldcg(&v->c2)}, x2));
        }
        acc = e3_warp_sum(acc);
        if (lane == 0) red[warp] = acc;
        __syncthreads();
        if (warp == 0) {
            acc = e3_warp_sum(lane < OPEN_WARPS ? red[lane] : e3_zero());
            if (lane == 0) sc->sum = e3_add(sc->sum, acc);
        }
    }
    if (warp == 0) {
        if (!cur[1]) wt.err |= TX_ERR_HINT_OVERFLOW;
        else wt.hints_len = hint_base + cur[0] * nwit;
        wtx_store(wt, a.tx);
        if (lane == 0) sc->counters[CTR_OPEN] = 0;
    }
}

int launch_open(const OpenArgs& a, cudaStream_t st) {
    if (a.q > (u32)MAX_QUERIES || (1u << a.fold) > (u32)MAX_DEPTH || a.nwit < 1 || a.nwit > (u32)MAX_WITNESSES) return -1;
    if (a.stir && (a.depth & ((1u << a.fold) - 1)) != 0) return -1;
    if (a.logN > OPEN_MAX_LOGN || a.ood_offset > MAX_OOD) return -1;
    // A row a warp of those that take the values, at most OPEN_CTAS.
    const u32 rows = OPEN_ROW_WARPS, ctas = std::min(OPEN_CTAS, std::max(1u, (a.q + rows - 1) / rows));
    k_open<<<ctas, OPEN_THREADS, 0, st>>>(a);
    count_launches(1);
    return 0;
}

}  // namespace wg
