// k_eqf_tc.cu -- the two weighted sums of EqFactoredProver's left phase
// (k_eqf.cu) over a base table p on the tensor cores:
//   inner sums   S[a]   = sum_b eq_r[b] p[a m + b]     (entry a, weights along p)
//   left folds   out[c] = sum_a e[a] p[a Lc + c]       (entry c, weights across p)
// Both are out[m] = sum_k W_k P(k, m) with Fp3 (or Fp) weights: a matrix
// product.  In 4-bit digits (tc.cuh) an entry's word is 16 rows of the first
// operand, the weights' components are 16 columns each of the second, K is
// the sum's index; a block takes 64 entries (eight accumulators of 128 x 48)
// and a range of K, exact in f32 up to 2^16 terms.  The integer pipes took
// three products per word and read the weights again for every entry (74 and
// 87 us at 2^24 entries, HBM alone 20).
//
// At 2^24 entries 47 and 41 us (four stages; three 48 and 43), two tables of
// that size in one launch 71: about 30 us are the loads (128 blocks, 16 KB a
// tile), a sixth the MMAs (eight of 48 columns a tile), the rest start and
// recombination.
// One block per SM: sixteen warps load p (16 bytes per lane and load, four
// tiles of 32 terms ahead), one warp loads the weights, one thread issues
// the MMAs; then the sixteen warps recombine the digits.
#include "tc.cuh"

namespace effsc {

constexpr int ET_M = 64, ET_K = 32;            // entries of a block, terms of a tile
constexpr int ET_LW = 16;
constexpr int ET_TPB = 32 * (ET_LW + 2);
constexpr int ET_S = 4, ET_AHEAD = 4;
constexpr u32 ET_ATOM = ET_K * 128;            // eight entries' digits
constexpr u32 ET_BYTES = 9 * ET_ATOM;          // eight atoms of p, one of the weights
constexpr u32 ET_SMEM = ET_S * ET_BYTES + 1024;

// The row of a tile's term q (stores of neighbouring or every other row of
// sixteen: no bank conflicts).
__device__ __forceinline__ u32 et_row(u32 q) { return q ^ ((q >> 3) & 1); }

// Blocks of M / 64 groups of entries of p, then as many of p2 (null: none).
// ALONG: P(k, m) = p[m s + k]; else P(k, m) = p[k s + m].  out: component c of
// entry m at part[3 (split M + m) + c], or without part (one split) at o[c][m].
template <bool ALONG, bool EW>
__global__ void __launch_bounds__(ET_TPB, 1) k_eqf_tc(const u64* p, const u64* p2, u64 stride, Tab3 w, u64 M, u64 K,
                                                      u32 splits, u64* part, u64* o0, u64* o1, u64* o2, TcWaits tw) {
    constexpr int NC = EW ? 3 : 1;
    extern __shared__ char et_dyn[];
    __shared__ u64 full[ET_S], empty[ET_S], done;
    __shared__ u32 s_tmem;
    char* stages = et_dyn + ((1024 - (smem_u32(et_dyn) & 1023)) & 1023);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        for (int s = 0; s < ET_S; s++) {
            mbar_init(&full[s], ET_LW + 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(&done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == ET_LW + 1) tc_alloc(&s_tmem, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const u32 tmem = s_tmem;
    const u32 split = blockIdx.x % splits;
    u64 m0 = (u64)(blockIdx.x / splits) * ET_M;
    if (m0 >= M) {                               // the second table's blocks
        m0 -= M;
        p = p2;
        part += 3 * M * splits;
    }
    const u64 kk = K / splits, k0 = split * kk;
    const u32 tiles = (u32)(kk / ET_K);
    bool abort = false;
    if (warp < ET_LW) {
        // two loads a tile: ALONG, entries 4 warp + 2 u and the next, 16 lanes
        // each; else term 2 warp + u of all 64 entries
        auto at = [&](u32 i, int u) {
            const u64 k = k0 + (u64)i * ET_K;
            return (const ulonglong2*)(ALONG ? p + (m0 + 4 * warp + 2 * u + (lane >> 4)) * stride + k + 2 * (lane & 15)
                                             : p + (k + 2 * warp + u) * stride + m0 + 2 * lane);
        };
        ulonglong2 v[ET_AHEAD][2];
#pragma unroll
        for (int q = 0; q < ET_AHEAD; q++)
            if ((u32)q < tiles)
#pragma unroll
                for (int u = 0; u < 2; u++) v[q][u] = __ldcs(at(q, u));
        for (u32 i0 = 0; i0 < tiles; i0 += ET_AHEAD) {
#pragma unroll
            for (int q = 0; q < ET_AHEAD; q++) {
                const u32 i = i0 + q;
                if (i >= tiles) break;
                const u32 s = i % ET_S;
                abort |= !mbar_wait_step(&empty[s], ((i / ET_S) & 1u) ^ 1u, tw.no_wait | abort);
                char* st = stages + s * ET_BYTES;
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    if (ALONG) {
                        const u32 m = 4 * warp + 2 * u + (lane >> 4), k = 2 * (lane & 15);
                        char* base = st + (m >> 3) * ET_ATOM;
                        *(uint4*)(base + swz128(et_row(k), m & 7)) = digits_of(v[q][u].x);
                        *(uint4*)(base + swz128(et_row(k + 1), m & 7)) = digits_of(v[q][u].y);
                    } else {
                        // even entries of one atom with odd ones of the next
                        const u32 k = et_row(2 * warp + u), m = 2 * lane, sel = (lane >> 2) & 1;
                        char* base = st + (m >> 3) * ET_ATOM;
                        *(uint4*)(base + swz128(k, (m & 7) + sel)) = digits_of(sel ? v[q][u].y : v[q][u].x);
                        *(uint4*)(base + swz128(k, (m & 7) + 1 - sel)) = digits_of(sel ? v[q][u].x : v[q][u].y);
                    }
                }
                if (i + ET_AHEAD < tiles)
#pragma unroll
                    for (int u = 0; u < 2; u++) v[q][u] = __ldcs(at(i + ET_AHEAD, u));
                fence_async_shared();
                __syncwarp();
                if (lane == 0) mbar_arrive(&full[s]);
            }
        }
    } else if (warp == ET_LW) {
        u64 x[2][NC];
#pragma unroll
        for (int q = 0; q < 2; q++)
            if ((u32)q < tiles)
#pragma unroll
                for (int c = 0; c < NC; c++) x[q][c] = w.c[c][k0 + (u64)q * ET_K + lane];
        for (u32 i0 = 0; i0 < tiles; i0 += 2) {
#pragma unroll
            for (int q = 0; q < 2; q++) {
                const u32 i = i0 + q;
                if (i >= tiles) break;
                const u32 s = i % ET_S;
                abort |= !mbar_wait_step(&empty[s], ((i / ET_S) & 1u) ^ 1u, tw.no_wait | abort);
                char* st = stages + s * ET_BYTES + 8 * ET_ATOM;
#pragma unroll
                for (int c = 0; c < NC; c++) *(uint4*)(st + swz128(et_row(lane), c)) = digits_of(x[q][c]);
                if (i + 2 < tiles)
#pragma unroll
                    for (int c = 0; c < NC; c++) x[q][c] = w.c[c][k0 + (u64)(i + 2) * ET_K + lane];
                fence_async_shared();
                __syncwarp();
                if (lane == 0) mbar_arrive(&full[s]);
            }
        }
    } else if (lane == 0) {
        for (u32 i = 0; i < tiles; i++) {
            const u32 s = i % ET_S;
            if (!mbar_wait_bounded(&full[s], (i / ET_S) & 1u)) { abort = true; break; }
            tc_fence_after();
            const u32 base = smem_u32(stages) + s * ET_BYTES;
            const u64 b = tc_desc(base + 8 * ET_ATOM, ET_ATOM, 1024);
#pragma unroll
            for (int m = 0; m < 8; m++)
                tc_mma_f8(tmem + 64 * m, tc_desc(base + m * ET_ATOM, ET_ATOM, 1024), b, tc_idesc(128, 16 * NC, true), i > 0);
            tc_commit(&empty[s]);
        }
        tc_commit(&done);
    }
    if (warp <= ET_LW || lane == 0) {
        if (!mbar_wait_bounded(&done, 0, 4000000000ULL)) abort = true;
    }
    __syncwarp();
    tc_fence_after();
    const bool bad = __syncthreads_or(abort);
    if (!bad && tiles && warp < ET_LW) {
#pragma unroll 1
        for (int e = 0; e < 2 * NC; e++) {
            const int blk = (warp >> 2) + 4 * (e / NC), c = e % NC;
            const u64 v = tc_row_sum(tmem + ((u32)(32 * (warp & 3)) << 16) + 64 * blk + 16 * c, lane);
            const u64 m = m0 + 8 * blk + 2 * (warp & 3) + (lane >> 4);
            if ((lane & 15) == 0) {
                if (part) part[3 * (split * M + m) + c] = v;
                else (c == 0 ? o0 : c == 1 ? o1 : o2)[m] = v;
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == ET_LW + 1) tc_dealloc(tmem, 512);
    if (bad && threadIdx.x == 0 && tw.status) *(volatile u32*)tw.status = EFFSC_STATUS_TIMEOUT;
}

// Blocks for M entries: splits of K until about a wave of blocks, at least
// two tiles each.
u32 eqf_tc_splits(u64 M, u64 K) {
    const u64 groups = M / ET_M;
    u64 s = 1;
    while (groups * s * 2 <= (u64)(max_grid() / 8) && K / (2 * s) >= 2 * ET_K) s *= 2;
    return (u32)s;
}
// Large sums over a base table that loads 16 bytes at a time.
bool eqf_tc_ok(bool along, u64 M, u64 K, u64 stride, const u64* p) {
    if (M % ET_M || K % ET_K || (stride & 1) || ((uintptr_t)p & 15) || M / ET_M > (1u << 20)) return false;
    return M * K >= (along ? EQF_TC_MIN_ROWS : EQF_TC_MIN) && K / eqf_tc_splits(M, K) <= 65536 && (K / eqf_tc_splits(M, K)) % ET_K == 0;
}
template <bool ALONG, bool EW>
static bool eqf_tc_inst(const u64* p, const u64* p2, u64 stride, Tab3 w, u64 M, u64 K, u32 splits, u64* part, u64* o0, u64* o1,
                        u64* o2, TcWaits tw, cudaStream_t s) {
    static std::atomic<uint64_t> configured{0};
    if (!tc_allow_smem(k_eqf_tc<ALONG, EW>, ET_SMEM, configured)) return false;
    k_eqf_tc<ALONG, EW><<<(int)((p2 ? 2 : 1) * (M / ET_M) * splits), ET_TPB, ET_SMEM, s>>>(p, p2, stride, w, M, K, splits, part, o0,
                                                                                       o1, o2, tw);
    return true;
}
bool launch_eqf_tc(bool along, bool ew, const u64* p, u64 stride, Tab3 w, u64 M, u64 K, u64* part, u64* o0, u64* o1, u64* o2,
                   TcWaits tw, cudaStream_t s) {
    const u32 splits = eqf_tc_splits(M, K);
    u64* pt = splits > 1 ? part : nullptr;
    bool ok;
    if (along) ok = ew ? eqf_tc_inst<true, true>(p, nullptr, stride, w, M, K, splits, pt, o0, o1, o2, tw, s)
                       : eqf_tc_inst<true, false>(p, nullptr, stride, w, M, K, splits, pt, o0, o1, o2, tw, s);
    else ok = ew ? eqf_tc_inst<false, true>(p, nullptr, stride, w, M, K, splits, pt, o0, o1, o2, tw, s)
                 : eqf_tc_inst<false, false>(p, nullptr, stride, w, M, K, splits, pt, o0, o1, o2, tw, s);
    if (ok && splits > 1) launch_eqf_sum(part, M, splits, ew ? 3 : 1, o0, o1, o2, s);
    return ok;
}
bool launch_eqf_tc_pair(bool along, bool ew, const u64* p, const u64* p2, u64 stride, Tab3 w, u64 M, u64 K, u64* part,
                        TcWaits tw, cudaStream_t s) {
    const u32 splits = eqf_tc_splits(2 * M, K);
    if (along) return ew && eqf_tc_inst<true, true>(p, p2, stride, w, M, K, splits, part, nullptr, nullptr, nullptr, tw, s);
    return ew ? eqf_tc_inst<false, true>(p, p2, stride, w, M, K, splits, part, nullptr, nullptr, nullptr, tw, s)
              : eqf_tc_inst<false, false>(p, p2, stride, w, M, K, splits, part, nullptr, nullptr, nullptr, tw, s);
}

}  // namespace effsc
