// k_tail.cu -- the last rounds of a Multilinear, InnerProduct or Coefficient
// (product of three Fp3 tables) proof in one thread block or one thread-block
// cluster.
//
// Once a prover's tables are small, a round costs far more in kernel
// boundaries (launch, grid-wide ticket, a lone last block running the
// transcript) than in arithmetic.  The tail kernel loads the tables into
// shared memory once (base tables embedded when the field is Fp3), then per
// round: folds with the previous challenge (new = lo + (hi - lo) r, reference
// src/inner_product_sumcheck.rs:143-176 and
// src/multilinear_sumcheck.rs:132-178), sums the round polynomial of the
// folded tables, and runs the transcript step (wire values, hook bytes,
// challenge squeeze) in warp 0.  After the last round the folded tables go
// back to global memory so that finalize / final_value and the post-state
// accessors see exactly what the per-round path would leave.  A batch
// launches one block per instance.
//
// What bounds it is one warp's latency: of 3.4 us a late round (InnerProduct
// over Fp3), 2.2 are the Keccak permutation, the rest the chain fold ->
// barrier -> sums -> barrier -> absorb, squeeze, reduce -> barrier.  n = 12:
// 110.8 us when a thread carried whole quadruples and the words were summed
// with shuffles, 74.8 in one block as split below, 66.6 in a cluster (whose
// two barriers a round cost less than the first rounds' folds on one SM), 58
// with the present permutation.
#include "round_common.cuh"

#include <atomic>
#include <cstring>

namespace effsc {

// How a round is split.  A late round is one block's latency, not its
// throughput: a few dozen entries, every step waiting for the one before.  So
// no thread carries a whole quadruple (36 products in a row): a fold with
// fewer entries than threads gives each thread one component of one folded
// entry (three products into one sum), the round polynomial gives each warp
// one row of products (a_k times b_0, b_1, b_2) of one of its two values, and
// a warp's sum takes three integer warp reductions (redux on 22-bit pieces)
// instead of five shuffle-and-add levels per word.  The challenge is left in
// shared memory together with its multiples by W.
constexpr int TAIL_TPB = 768;        // 24 warps: a multiple of the 6 components of two Fp3 values
constexpr int TAIL_NW = TAIL_TPB / 32;

// Index i of a table of 2^lg entries with its lg bits reversed.  An LSB
// prover's table held in this order makes its folds (2j, 2j+1) -> j MSB
// folds (p, p + L/2) -> p, in place, with entry j of every later length at
// the reversed position again; so the LSB tail is the MSB tail on a
// bit-reversed layout, reversed back when the tables are written out.
__device__ __forceinline__ u32 tail_rev(u32 i, u32 lg) { return lg ? __brev(i) >> (32 - lg) : 0; }
// The entry that step i of an LSB load takes: neighbouring lanes four entries
// in a row (a sector), eight such runs an eighth of the table apart, which
// are neighbours once reversed.  In order, a warp's reversed stores would all
// meet in one bank (InnerProduct over Fp3, the tail from 2^16 entries: 127 ->
// 123 us; a whole proof of 2^16: 138 -> 131).
__device__ __forceinline__ u32 tail_spread(u32 i, u32 lg) {
    return lg < 5 ? i : ((i >> 2 & 7) << (lg - 3)) | (i >> 5 << 2) | (i & 3);
}
__device__ __forceinline__ u32 tail_lg(u32 n) { return n > 1 ? 31 - __clz(n) : 0; }

constexpr int TAIL_MAX_CS = 16;
// Shared state of a tail block.
struct TailShared {
    uint4 part[3 * TAIL_NW];           // the warps' sums, in 22-bit pieces
    u64 chal[5];                       // W r1, W r2, r0, r1, r2 of the last challenge r
    u64 tot[9];                        // wire values, component c of value e at 3 e + c
    u64 raw[3];
    __align__(8) uint8_t scr[64];
    u64 cred[TAIL_MAX_CS][9];          // (cluster kernel, CTA 0) every CTA's sums
};

// Where a tail's tables are: component c of table t, entry i at
// sm[(t FW + c) stride + off + i].  A fold writes the half of its rows that
// the table does not occupy (off alternates between 0 and stride / 2), so
// that threads may share an entry; only a table that fills its rows is
// folded in place, by one thread per entry.
struct TailTab {
    u64* sm;
    u32 stride, off, len;
};

// Component c of lo + (hi - lo) r; ch = the prepared challenge.
template <int FW>
__device__ __forceinline__ u64 tail_fold_comp(const u64* row0, u32 stride, u32 j, u32 half, int c, const u64* ch) {
    AccF<FOLD_FORM> s;
    s.from(row0[c * stride + j]);
    // c0 = d0 r0 + d1 W r2 + d2 W r1, c1 = d0 r1 + d1 r0 + d2 W r2, c2 = d0 r2 + d1 r1 + d2 r0
    u64 d[FW];
#pragma unroll
    for (int k = 0; k < FW; k++) d[k] = gl_sub(row0[k * stride + j + half], row0[k * stride + j]);
#pragma unroll
    for (int k = 0; k < FW; k++) s.mac(d[k], ch[2 + c - k]);
    return s.reduce();
}

// Fold every table (pairs j, j + len/2).  `base`: the entries' components 1
// and 2 are zero (tables given in Fp, Fp3 challenges).  put(t, c, j, value)
// sees the folded entries too.  In place when out == T.off.
template <int NT, int FW, class Put>
__device__ __forceinline__ void tail_fold(const TailTab& T, u32 out, bool base, const u64* ch, Put put) {
    const u32 half = T.len >> 1;
    if (FW == 3 && (out == T.off || NT * half >= TAIL_TPB)) {
        // a whole entry per thread
        Mul3 m;
        m.w1 = ch[0]; m.w2 = ch[1]; m.m0 = ch[2]; m.m1 = ch[3]; m.m2 = ch[4];
        const u32 lg = tail_lg(half);
        for (u32 i = threadIdx.x; i < NT * half; i += TAIL_TPB) {
            const int t = NT > 1 ? i >> lg : 0;
            const u32 j = i - t * half;
            const u64* row = T.sm + t * 3 * T.stride + T.off;
            u64* dst = T.sm + t * 3 * T.stride + out;
            F3 lo, hi, v;
            lo.c0 = row[j]; hi.c0 = row[j + half];
            if (base) {
                lo.c1 = lo.c2 = hi.c1 = hi.c2 = 0;
                v = f3_fold<false, true>(lo, hi, m);
            } else {
                lo.c1 = row[T.stride + j]; lo.c2 = row[2 * T.stride + j];
                hi.c1 = row[T.stride + j + half]; hi.c2 = row[2 * T.stride + j + half];
                v = f3_fold<true, true>(lo, hi, m);
            }
            dst[j] = v.c0; dst[T.stride + j] = v.c1; dst[2 * T.stride + j] = v.c2;
            put(t, 0, j, v.c0); put(t, 1, j, v.c1); put(t, 2, j, v.c2);
        }
        return;
    }
    // one component of one entry per thread and step, j fastest
    const u32 lg = tail_lg(half);
    for (u32 i = threadIdx.x; i < NT * FW * half; i += TAIL_TPB) {
        const u32 r = i >> lg;                        // t FW + c
        const int t = NT > 1 ? r / FW : 0, c = (int)r - t * FW;
        const u32 j = i & (half - 1);
        const u64 v = tail_fold_comp<FW>(T.sm + t * FW * T.stride + T.off, T.stride, j, half, c, ch);
        T.sm[r * T.stride + out + j] = v;
        put(t, c, j, v);
    }
}

// The warps' work on the round polynomial, NWIRE values of FW components:
//   InnerProduct: q0 = sum a_lo b_lo, qinf = sum (a_hi - a_lo)(b_hi - b_lo)
//   (src/provers/inner_product.rs:94-103); Multilinear: the wire is
//   s0 = sum lo alone (src/provers/multilinear.rs:52-61).
// The warps divide into roles with WPR warps each, slot s of a role taking the
// entries 32 s + lane, + 32 WPR, ...:
//   TERM  (IP over Fp3, at most 32 pairs) one product: x_k y_m of value
//         `which`, m = (c - k) mod 3, its y times W where the index wraps;
//   ROW   (IP over Fp3) x_k with all three y_m;
//   VALUE (Fp, or Fp3 before base tables' first fold) a whole value; ML over
//         Fp3: one component of it.
// CoefficientProver's product of three Fp3 tables (POL_C3W): h(0), h(inf) and
// h(2), sums of a product of three each (src/provers/coefficient.rs:272-294);
// a role is a value, a lane a pair.
// Every sum goes to sh.part, those of a wire word next to each other, wire word `word` is the sum of its TERMS x slots entries.
template <int POL, int FW>
struct TailRoles {
    static constexpr int NWIRE = POL == POL_ML ? 1 : POL == POL_C3W ? 3 : 2;
    static constexpr int N = NWIRE * FW;                  // wire words
    static constexpr bool ROWS = POL == POL_IP && FW == 3;
    static constexpr int WPR = TAIL_NW / N, WPR_BASE = TAIL_NW / NWIRE;
};

// A round's sums over the current tables into sh.part; returns how many
// slots of each role held entries.
template <int POL, int FW>
__device__ __forceinline__ u32 tail_eval(const TailTab& T, bool base, TailShared& sh) {
    using R = TailRoles<POL, FW>;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const u32 half = T.len > 1 ? T.len >> 1 : 1;         // a single entry feeds h(0) alone
    const u64* a = T.sm + T.off;
    const u64* b = a + FW * T.stride;
    if (R::ROWS && !base && half <= 32) {
        // TERM
        const int word = warp / 3, k = warp - 3 * word, which = word >= 3, c = word - 3 * which;
        if (word < 6) {
            const int m = c - k + (k > c ? 3 : 0);
            u64 v = 0;
            if (lane < (int)half && (T.len > 1 || !which)) {
                const u64 *pa = a + k * T.stride + lane, *pb = b + m * T.stride + lane;
                u64 x = pa[0], y = pb[0];
                if (which) { x = gl_sub(pa[half], x); y = gl_sub(pb[half], y); }
                if (k > c) y = gl_mul_w(y);
                v = gl_mul(x, y);
            }
            __syncwarp();
            const uint4 p = warp_sum_pieces(v);
            if (lane == 0) sh.part[warp] = p;
        }
        return 1;
    }
    const bool whole = base || POL == POL_C3W;          // a role is a value, not a component or row of one
    const u32 wpr = whole ? R::WPR_BASE : R::WPR;
    const u32 role = whole ? warp / R::WPR_BASE : warp / R::WPR, slot = warp - role * wpr;
    const u32 slots = min(wpr, (half + 31) >> 5);
    if (slot >= slots) return slots;
    const u32 j0 = slot * 32 + lane, step = 32 * wpr;
    if constexpr (POL == POL_C3W) {
        // role = a point of the wire: lo (0), hi - lo (infinity), 2 hi - lo (2)
        ProdAcc<true, true> s;
        s.init();
        for (u32 j = j0; j < half; j += step) {
            F3 x[3];
#pragma unroll
            for (int t = 0; t < 3; t++) {
                const u64* q = a + 3 * t * T.stride + j;
                x[t] = f3_make(q[0], q[T.stride], q[2 * T.stride]);
                if (role) {
                    const F3 hi = f3_make(q[half], q[T.stride + half], q[2 * T.stride + half]);
                    x[t] = f3_sub<true>(hi, x[t]);
                    if (role == 2) x[t] = f3_add<true>(hi, x[t]);
                }
            }
            s.mac(f3_mul<true, true>(x[0], x[1]), x[2]);
        }
        const F3 v = s.result();
        const uint4 p0 = warp_sum_pieces(v.c0), p1 = warp_sum_pieces(v.c1), p2 = warp_sum_pieces(v.c2);
        if (lane == 0) {
            uint4* d = sh.part + 3 * role * slots + slot;
            d[0] = p0;
            d[slots] = p1;
            d[2 * slots] = p2;
        }
        return slots;
    }
    if (R::ROWS && !base) {
        const u32 which = role >= 3, k = role - 3 * which;
        AccF<0> s[3];
#pragma unroll
        for (int o = 0; o < 3; o++) s[o].zero();
        const u64* ak = a + k * T.stride;
        for (u32 j = j0; j < half; j += step) {
            u64 x = ak[j], y[3];
#pragma unroll
            for (int o = 0; o < 3; o++) y[o] = b[o * T.stride + j];
            if (which) {
                x = gl_sub(ak[j + half], x);
#pragma unroll
                for (int o = 0; o < 3; o++) y[o] = gl_sub(b[o * T.stride + j + half], y[o]);
            }
#pragma unroll
            for (int o = 0; o < 3; o++) s[o].mac(x, y[o]);
        }
#pragma unroll
        for (int o = 0; o < 3; o++) {
            const bool wrap = k + o >= 3;
            u64 v = s[o].reduce();
            if (wrap) v = gl_mul_w(v);
            const uint4 p = warp_sum_pieces(v);
            // wire word 3 which + (k + o) mod 3, its term k
            if (lane == 0) sh.part[((3 * which + k + o - (wrap ? 3 : 0)) * 3 + k) * slots + slot] = p;
        }
        return slots;
    }
    Acc s = acc_zero();
    for (u32 j = j0; j < half; j += step) {
        if (POL == POL_ML) {
            acc_add64(s, a[role * T.stride + j]);
        } else {
            u64 x = a[j], y = b[j];
            if (role) {
                x = T.len > 1 ? gl_sub(a[j + half], x) : 0;
                y = T.len > 1 ? gl_sub(b[j + half], y) : 0;
            }
            acc_mac(s, x, y);
        }
    }
    const uint4 p = warp_sum_pieces(acc_reduce(s));
    if (lane == 0) sh.part[role * slots + slot] = p;
    return slots;
}
// Wire word (which FW + c) from sh.part, in that lane; 0 in the others.
template <int POL, int FW>
__device__ __forceinline__ u64 tail_total(const TailShared& sh, int lane, bool base, u32 slots) {
    using R = TailRoles<POL, FW>;
    u64 v = 0;
    if (lane < R::N && !(base && lane % FW)) {
        const u32 n = R::ROWS && !base ? 3 * slots : slots;
        const uint4* q = sh.part + (base ? lane / FW : lane) * n;
        uint4 s = q[0];
        for (u32 i = 1; i < n; i++) {
            const uint4 p = q[i];
            s.x += p.x; s.y += p.y; s.z += p.z;
        }
        v = join_pieces(s);
    }
    __syncwarp();
    return v;
}

// The transcript of a tail, in warp 0.
struct TailTx {
    WarpTx w;
    TxStream s;
};
template <int NW>
__device__ __forceinline__ void tail_tx_init(TailTx& x, const TailArgs& a, int lane) {
    x.w = tx_load((const DevTranscript*)a.tx, lane);
    x.s = tx_stream(NW, a.hook, a.hook_len, lane);
}
// The wire values (word FW e + c in that lane) times the scalar, by a whole warp.
template <int POL, int FW>
__device__ __forceinline__ u64 tail_scale(u64 wire, const TailArgs& a, int lane) {
    constexpr int NW = TailRoles<POL, FW>::N;
    if (FW == 1) return lane < NW ? gl_mul(wire, a.scalar[0][0]) : 0;
    const int e = 3 * (lane / 3) < NW ? 3 * (lane / 3) : 0;
    const F3 x = f3_make(shfl64(wire, e), shfl64(wire, e + 1), shfl64(wire, e + 2));
    const F3 y = f3_mul<true, true>(x, ld_scalar(a.scalar));
    return lane >= NW ? 0 : lane % 3 == 0 ? y.c0 : lane % 3 == 1 ? y.c1 : y.c2;
}
// The transcript step of a round: send the wire values (word i of them in
// lane i), absorb the hook, squeeze the challenge into sh.chal, prepared.
template <int POL, int FW>
__device__ __forceinline__ void tail_transcript(TailTx& x, u64 wire, const TailArgs& a, TailShared& sh) {
    constexpr int NW = TailRoles<POL, FW>::N;
    const int lane = threadIdx.x & 31;
    if (POL == POL_IP && a.scalar[0]) wire = tail_scale<POL, FW>(wire, a, lane);
    if (lane < NW) sh.tot[FW == 3 ? lane : 3 * lane] = wire;
    const u64 r = tx_step(x.w, x.s, NW, FW, wire, a.hook, a.hook_len, lane, sh.tot, sh.raw, sh.scr);
    if (lane < 3) sh.chal[2 + lane] = r;
    if (FW == 3 && (lane == 1 || lane == 2)) sh.chal[lane - 1] = gl_mul_w(r);
}
// Round k's wire values and challenge into the proof, by the last warp after
// the barrier that publishes them (the next round changes them two barriers
// later).
template <int POL, int FW>
__device__ __forceinline__ void tail_record(const TailArgs& a, u32 k, const TailShared& sh) {
    constexpr u32 NW3 = 3 * TailRoles<POL, FW>::NWIRE;
    const u32 i = threadIdx.x - (TAIL_TPB - 32);
    if (i < NW3) a.proof_wire[k * NW3 + i] = FW == 3 || i % 3 == 0 ? sh.tot[i] : 0;
    else if (i >= 16 && i < 19) a.proof_chal[3 * k + i - 16] = sh.chal[i - 14];
}

// The challenge before the first round, prepared (or zeros).
template <int FW>
__device__ __forceinline__ void tail_first_challenge(const TailArgs& a, TailShared& sh) {
    if (threadIdx.x < 3) {
        const u64 r = a.first_fold ? a.chal_in[threadIdx.x] : 0;
        sh.chal[2 + threadIdx.x] = r;
        if (threadIdx.x) sh.chal[threadIdx.x - 1] = gl_mul_w(r);
    }
}

// The next fold's destination: the half of the rows the table is not in.
__device__ __forceinline__ u32 tail_next_off(const TailTab& T) {
    return T.len == T.stride ? T.off : T.off ? 0 : T.stride >> 1;
}

// Rounds k0 .. a.nrounds-1 in one block, then the transcript state, the
// runner's finalize fold, the read-back entries and the folded tables.
template <int POL, int FW>
__device__ __forceinline__ void tail_loop(TailTab T, u32 k0, bool fold, bool base, const TailArgs& a, TailTx& x,
                                          TailShared& sh) {
    constexpr int NT = Policy<POL, 0>::NT;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (u32 k = k0; k < a.nrounds; k++) {
        if (fold) {
            const u32 out = tail_next_off(T);
            tail_fold<NT, FW>(T, out, base, sh.chal, [](int, int, u32, u64) {});
            T.off = out;
            T.len >>= 1;
            base = false;
            __syncthreads();
        }
        const u32 slots = tail_eval<POL, FW>(T, base, sh);
        __syncthreads();
        if (warp == 0) tail_transcript<POL, FW>(x, tail_total<POL, FW>(sh, lane, base, slots), a, sh);
        __syncthreads();
        tail_record<POL, FW>(a, k, sh);
        fold = true;
    }
    if (warp == 0) tx_store((DevTranscript*)a.tx, x.w, lane);
    if (a.final_fold && T.len >= 2) {
        // SumcheckProver::finalize with the last challenge: one MSB fold
        // (src/inner_product_sumcheck.rs:143-176, src/multilinear_sumcheck.rs:132-178)
        const u32 out = tail_next_off(T);
        tail_fold<NT, FW>(T, out, base, sh.chal, [](int, int, u32, u64) {});
        T.off = out;
        T.len >>= 1;
        __syncthreads();
    }
    if (a.first_out && threadIdx.x < 12) {
        const int t = threadIdx.x / 3, c = threadIdx.x % 3;
        a.first_out[threadIdx.x] = (t < NT && c < FW) ? T.sm[(t * FW + c) * T.stride + T.off] : 0;
    }
    // write back the tables after the last fold (LSB: from the reversed layout)
    if (a.out[0][0]) {
        const u32 lg = tail_lg(T.len);
        for (int t = 0; t < NT; t++)
            for (int c = 0; c < FW; c++) {
                const u64* src = T.sm + (t * FW + c) * T.stride + T.off;
                u64* dst = a.out[t][c];
                for (u32 i = threadIdx.x; i < T.len; i += TAIL_TPB) dst[i] = src[a.lsb ? tail_rev(i, lg) : i];
            }
    }
}

// One block: rows of the starting length.  Warp 0 keeps the transcript state
// in registers for the whole tail.
template <int POL, int FW>
__device__ __forceinline__ void tail_body(const TailArgs& a) {
    extern __shared__ __align__(16) u64 sm[];
    constexpr int NT = Policy<POL, 0>::NT;
    __shared__ TailShared sh;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const u32 L0 = (u32)a.L, lg0 = tail_lg(L0);
    for (int t = 0; t < NT; t++)
        for (int c = 0; c < FW; c++) {
            const u64* src = (c == 0 || ((a.in_ext >> t) & 1u)) ? a.in[t][c] : nullptr;
            u64* dst = sm + (t * FW + c) * L0;
            if (a.lsb)
                for (u32 i = threadIdx.x; i < L0; i += TAIL_TPB) {
                    const u32 j = tail_spread(i, lg0);
                    dst[tail_rev(j, lg0)] = src ? src[j] : 0;
                }
            else
                for (u32 i = threadIdx.x; i < L0; i += TAIL_TPB) dst[i] = src ? src[i] : 0;
        }
    tail_first_challenge<FW>(a, sh);
    TailTx x;
    if (warp == 0) tail_tx_init<TailRoles<POL, FW>::N>(x, a, lane);
    __syncthreads();
    TailTab T{sm, L0, 0, L0};
    tail_loop<POL, FW>(T, 0, a.first_fold != 0, FW == 3 && a.in_ext == 0, a, x, sh);
}

// ---- cluster tail ---------------------------------------------------------
// Tables up to CS times one block's capacity, and smaller ones whose first
// rounds are worth sharing: a thread-block cluster of CS CTAs holds them in
// distributed shared memory.  MSB: CTA c holds the groups of G consecutive
// entries whose group index is c mod CS: entry k with (k / G) mod CS = c at
// local index (k / (G CS)) G + k mod G; the slices load as whole sectors
// (G = 16: lines), and pairs (k, k + L/2) are local pairs (j, j + L/(2 CS))
// while L/2 is a multiple of G CS.  LSB: CTA c holds the entries c Ll ..
// (c + 1) Ll - 1 bit-reversed among themselves, so its first log2(Ll) folds
// are local too.  Each CTA folds and evaluates its slice exactly as the
// one-block tail does; the CTAs' sums meet in CTA 0 (distributed shared
// memory stores), which runs the transcript step and writes the challenge
// back into every CTA.  Fold log2(CS) + 1 also writes the table (now half a
// slice long) into CTA 0's free half, which finishes the proof alone.  Every
// CTA passes the same cluster barriers, two per round.
// Global index of local entry j of CTA c.
__device__ __forceinline__ u32 cl_global(u32 j, u32 c, u32 cs_log, u32 g_log) {
    return ((((j >> g_log) << cs_log) + c) << g_log) + (j & ((1u << g_log) - 1));
}
__device__ __forceinline__ u32 cluster_rank() {
    u32 r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Store v at the shared-memory location p of CTA `rank` in the cluster.
__device__ __forceinline__ void dsmem_st(const void* p, u32 rank, u64 v) {
    u32 remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(p)), "r"(rank));
    asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(remote), "l"(v) : "memory");
}

template <int POL, int FW>
__global__ void __launch_bounds__(TAIL_TPB, 1) k_tail_cluster(TailArgs a, u32 cs_log, u32 g_log) {
    extern __shared__ __align__(16) u64 sm[];
    constexpr int NT = Policy<POL, 0>::NT;
    constexpr int NW = TailRoles<POL, FW>::N;
    __shared__ TailShared sh;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const u32 CS = 1u << cs_log, rank = cluster_rank();
    chain_enter();
    const u32 Ll = (u32)(a.L >> cs_log);     // slice length (row stride)
    const u32 lgl = tail_lg(Ll);
    // this CTA's slice; base tables are embedded when the field is Fp3
    for (int t = 0; t < NT; t++)
        for (int c = 0; c < FW; c++) {
            const u64* src = (c == 0 || ((a.in_ext >> t) & 1u)) ? a.in[t][c] : nullptr;
            u64* dst = sm + (t * FW + c) * Ll;
            if (a.lsb)
                for (u32 i = threadIdx.x; i < Ll; i += TAIL_TPB) {
                    const u32 j = tail_spread(i, lgl);
                    dst[tail_rev(j, lgl)] = src ? src[rank * Ll + j] : 0;
                }
            else
                for (u32 j = threadIdx.x; j < Ll; j += TAIL_TPB) dst[j] = src ? src[cl_global(j, rank, cs_log, g_log)] : 0;
        }
    tail_first_challenge<FW>(a, sh);
    TailTx x;
    if (rank == 0 && warp == 0) tail_tx_init<NW>(x, a, lane);
    cluster_sync_all();   // every CTA is running before any remote store
    TailTab T{sm, Ll, 0, Ll};
    bool base = FW == 3 && a.in_ext == 0, fold = a.first_fold != 0;
    u32 gather = 0, left = cs_log + 1;       // folds to the hand-over
    u32 k = 0;
    for (; left; k++) {
        if (fold) {
            u32 out = tail_next_off(T);
            if (--left) {
                tail_fold<NT, FW>(T, out, base, sh.chal, [](int, int, u32, u64) {});
            } else {
                // the whole folded table goes to the free half of CTA 0's rows,
                // at its global (LSB: globally bit-reversed) index; the slice
                // itself is folded next to its source, into the half that holds
                // it (Ll / CS entries there, half of that written, CS >= 4)
                gather = out;
                out = T.off + T.len;
                const u32 rrev = tail_rev(rank, cs_log);
                tail_fold<NT, FW>(T, out, base, sh.chal, [&](int t, int c, u32 j, u64 v) {
                    const u32 g = a.lsb ? (j << cs_log) + rrev : cl_global(j, rank, cs_log, g_log);
                    dsmem_st(sm + (t * FW + c) * Ll + gather + g, 0, v);
                });
            }
            T.off = out;
            T.len >>= 1;
            base = false;
            __syncthreads();
        }
        fold = true;
        const u32 slots = tail_eval<POL, FW>(T, base, sh);
        __syncthreads();
        if (warp == 0) {
            const u64 v = tail_total<POL, FW>(sh, lane, base, slots);
            if (lane < NW) dsmem_st(&sh.cred[rank][lane], 0, v);
        }
        cluster_sync_all();   // all CTAs' sums (and at the hand-over the table) are in CTA 0
        if (rank == 0 && warp == 0) {
            u64 wire = 0;
            if (lane < NW) {
                Acc v = acc_zero();
                for (u32 c = 0; c < CS; c++) acc_add64(v, sh.cred[c][lane]);
                wire = acc_reduce(v);
            }
            tail_transcript<POL, FW>(x, wire, a, sh);
            __syncwarp();
            if (lane >= 1 && (u32)lane < CS)
                for (int c = 0; c < 5; c++) dsmem_st(&sh.chal[c], (u32)lane, sh.chal[c]);
        }
        cluster_sync_all();   // the challenge is in every CTA
        if (rank == 0) tail_record<POL, FW>(a, k, sh);
    }
    if (rank != 0) return;    // no remote access to this CTA follows
    T.off = gather;
    T.len = Ll >> 1;
    tail_loop<POL, FW>(T, k, true, false, a, x, sh);
}

template <int POL, int FW>
__global__ void __launch_bounds__(TAIL_TPB, 1) k_tail_one(TailArgs a) {
    chain_enter();
    tail_body<POL, FW>(a);
}
template <int POL, int FW>
__global__ void __launch_bounds__(TAIL_TPB, 1) k_tail_many(const TailArgs* args) { tail_body<POL, FW>(args[blockIdx.x]); }

u64 tail_max_len(int pol, int fw, u64 smem_cap) {
    const u64 per = (u64)pol_ntables(pol) * fw * sizeof(u64);
    u64 L = 1;
    while (2 * L * per <= smem_cap) L *= 2;
    return L;
}

template <int POL, int FW>
static bool tail_inst(const TailArgs* dev_args, const TailArgs* one, u32 n, u64 smem_len, cudaStream_t s) {
    const size_t bytes = (size_t)pol_ntables(POL) * FW * smem_len * sizeof(u64);
    if (bytes > TAIL_SMEM_CAP) return false;
    if (one) {
        cudaFuncSetAttribute(k_tail_one<POL, FW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TAIL_SMEM_CAP);
        return launch_dep(k_tail_one<POL, FW>, 1, TAIL_TPB, bytes, s, *one);
    } else {
        cudaFuncSetAttribute(k_tail_many<POL, FW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TAIL_SMEM_CAP);
        k_tail_many<POL, FW><<<n, TAIL_TPB, bytes, s>>>(dev_args);
    }
    return true;
}

template <int POL, int FW>
static bool tail_cluster_inst(const TailArgs& a, u32 cs_log, u32 g_log, cudaStream_t s) {
    const u32 CS = 1u << cs_log;
    const size_t bytes = (size_t)pol_ntables(POL) * FW * (a.L >> cs_log) * sizeof(u64);
    if (bytes > TAIL_SMEM_CAP || CS > (u32)TAIL_MAX_CS) return false;
    cudaFuncSetAttribute(k_tail_cluster<POL, FW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TAIL_SMEM_CAP);
    if (CS > 8) cudaFuncSetAttribute(k_tail_cluster<POL, FW>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(CS, 1, 1);
    cfg.blockDim = dim3(TAIL_TPB, 1, 1);
    cfg.dynamicSmemBytes = bytes;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CS;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_on(true) ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, k_tail_cluster<POL, FW>, a, cs_log, g_log) == cudaSuccess;
}

// Largest cluster the device runs for the cluster tail (8 or 16 CTAs of
// TAIL_SMEM_CAP bytes each; 0 when none fits).
u32 tail_cluster_max(void) {
    static std::atomic<int> cached[64];   // per device: 0 unknown, else size + 1
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    std::atomic<int>& slot = cached[dev & 63];
    int v = slot.load();
    if (v > 0) return (u32)(v - 1);
    v = 0;
    for (u32 cs : {16u, 8u}) {
        cudaFuncSetAttribute(k_tail_cluster<POL_ML, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TAIL_SMEM_CAP);
        if (cs > 8 && cudaFuncSetAttribute(k_tail_cluster<POL_ML, 3>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
            cudaGetLastError();
            continue;
        }
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(cs, 1, 1);
        cfg.blockDim = dim3(TAIL_TPB, 1, 1);
        cfg.dynamicSmemBytes = TAIL_SMEM_CAP;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = cs;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, k_tail_cluster<POL_ML, 3>, &cfg) == cudaSuccess && n > 0) { v = (int)cs; break; }
        cudaGetLastError();
    }
    slot.store(v + 1);
    return (u32)v;
}

bool launch_tail_cluster(int pol, int fw, const TailArgs& a, u32 cs_log, u32 g_log, cudaStream_t s) {
    switch (pol * 4 + fw) {
    case POL_ML * 4 + 1: return tail_cluster_inst<POL_ML, 1>(a, cs_log, g_log, s);
    case POL_ML * 4 + 3: return tail_cluster_inst<POL_ML, 3>(a, cs_log, g_log, s);
    case POL_IP * 4 + 1: return tail_cluster_inst<POL_IP, 1>(a, cs_log, g_log, s);
    case POL_IP * 4 + 3: return tail_cluster_inst<POL_IP, 3>(a, cs_log, g_log, s);
    case POL_C3W * 4 + 3: return tail_cluster_inst<POL_C3W, 3>(a, cs_log, g_log, s);
    default: return false;
    }
}

// The split of a tail over a cluster: as many CTAs as the device runs and the
// slices allow (at least 4), groups of 16 entries where the pairs stay in
// their CTA to the hand-over, else of 4 (which also leaves LSB slices of
// at least 4 entries there).
bool tail_cluster_split(int pol, int fw, u64 L, u32 rounds, bool first_fold, u32* cs_log, u32* g_log) {
    if (L < TAIL_CLUSTER_MIN || (L & (L - 1)) || L > (1u << 30)) return false;
    const u64 cap = tail_max_len(pol, fw, TAIL_SMEM_CAP);
    for (u32 lg = 4; lg >= 2; lg--) {
        const u64 cs = 1ull << lg;
        if (cs > tail_cluster_max() || L / cs > cap) continue;
        const u64 last = L >> (lg + 2);          // half of the table handed over
        if (last % (4 * cs) != 0) continue;
        const u32 folds = rounds - (first_fold ? 0 : 1);
        if (rounds < 1 || folds < lg + 1 || folds >= 63 || (L >> folds) < 2) continue;
        *cs_log = lg;
        *g_log = last % (16 * cs) == 0 ? 4 : 2;
        return true;
    }
    return false;
}

bool launch_tail(int pol, int fw, const TailArgs* dev_args, const TailArgs* one, u32 n, u64 smem_len, cudaStream_t s) {
    if (!n) return true;
    switch (pol * 4 + fw) {
    case POL_ML * 4 + 1: return tail_inst<POL_ML, 1>(dev_args, one, n, smem_len, s);
    case POL_ML * 4 + 3: return tail_inst<POL_ML, 3>(dev_args, one, n, smem_len, s);
    case POL_IP * 4 + 1: return tail_inst<POL_IP, 1>(dev_args, one, n, smem_len, s);
    case POL_IP * 4 + 3: return tail_inst<POL_IP, 3>(dev_args, one, n, smem_len, s);
    case POL_C3W * 4 + 3: return tail_inst<POL_C3W, 3>(dev_args, one, n, smem_len, s);
    default: return false;
    }
}

}  // namespace effsc
