// k_gram.cu -- the first pass of the InnerProduct start (rounds 0 .. NV - 1,
// NV = 3 or 4) on the tensor cores.
//
// Write a group of 2^NV entries of a table as v(t_0, .., t_{NV-1}), t_i the
// variable bound in round i, and G_ij = sum over the groups of x_i y_j.  Folded
// with r_0 .. r_{k-1} (src/inner_product_sumcheck.rs:143-176) a table's group
// is sum_p w_p v(p, .), w the eq weights of the challenges, so round k's wire
// (src/provers/inner_product.rs:94-103)
//   q0   = sum_{p, p'} w_p w_p' sum_s G[p 0 s][p' 0 s]
//   qinf = sum_{p, p'} w_p w_p' sum_s (G[p1s][p'1s] - G[p1s][p'0s] - G[p0s][p'1s] + G[p0s][p'0s])
// needs nothing of the tables but G: one pass, a Gram matrix -- a matrix
// product with the groups as its inner dimension.  Split into 4-bit digits
// (tc.cuh) a group of a table is 16 x 2^NV bytes, and G's digit sums are one
// 128 x 128 (256 x 256) product, exact in f32 up to 74565 groups per
// accumulator.
//
// One block per SM.  Sixteen warps load the tables (each lane 16 bytes at a
// time, GR_AHEAD tiles ahead, in registers), split the words and store the
// digit rows; a stage is a tile of 128 groups of both tables, the M / N index
// contiguous, as both operands of tcgen05.mma take it.  One thread of a
// seventeenth warp issues a stage's MMAs as soon as the stage is full and
// commits it empty.  At the end a warp per 32 accumulator rows reads them out
// of tensor memory and recombines the digits into G mod p; the last block to
// finish adds up the blocks' and runs the rounds' transcript steps.
//
// Bound: HBM (16 bytes per entry of the tables).  Per group of eight entries
// an SM spends about 1.8 cycles on the ALU (96 mask and shift instructions
// against the 530 of 26 products with their differences), 4 on shared memory
// (256 bytes written, 256 read by the MMAs) and 2 on the tensor core (NV = 4:
// twice that), where the tables take 5.8 cycles to arrive.
// Measured, n = 26: rounds 0-2 in 310 us on the integer pipes, 215 us here
// with NV = 3, rounds 0-3 in 236 us with NV = 4 (~30 us of it the last block's
// reduction and the four transcript steps) and 210 us with each tile asked into
// L2 two tiles before its register loads (four ahead 216, eight 241) and
// streaming loads, 206 with two stages instead of three (more L1 for the loads).
#include "ip012.cuh"
#include "residency.h"
#include "tc.cuh"
#include "tc_plan.h"

namespace effsc {

constexpr int GR_LW = 16;                     // loading warps
constexpr int GR_TPB = 32 * (GR_LW + 1);
constexpr u64 GR_LIMIT_NS = tc_wait_ns(false), GR_HOST_LIMIT_NS = tc_wait_ns(true);
constexpr u32 GR_MAX_TILES = 65536 / 128;     // tiles per accumulator: 2^16 groups (2^16 * 225 < 2^24)

template <bool LSB, int NV>
struct Gram {
    using Tile = TcTile<LSB, NV>;
    static constexpr int V = 1 << NV;
    static constexpr int UPW = Tile::UNITS / GR_LW;       // units per warp and tile
    static constexpr int AHEAD = NV == 3 ? 4 : 2;         // tiles in flight in registers
    static constexpr int S = NV == 3 ? 4 : 2;             // stages of 32 (64) KB: the rest is L1 for the loads in flight
    static constexpr u32 SMEM = S * Tile::BYTES + 1024;
    static constexpr u32 COLS = NV == 3 ? 128 : 512;      // tensor memory
    static constexpr int NQ = ((1 << (2 * NV)) - 1) / 3;  // entries of the rounds' matrices
    struct Shared {
        u64 full[S], empty[S], done;
        u32 tmem;
        int last;
        u64 g[V * V];
        u64 fin[2][V * V];
        u64 q[2][NQ];             // round k at (4^k - 1) / 3: q0's and qinf's matrix over (p, p')
        u64 w[V / 2][3];          // the weights w_p
        u64 v[2][V / 2][3];
        u64 tot[6], raw[3];
        __align__(8) uint8_t scr[64];
    };
};

// The accumulators -> G, a warp per 32 rows (two of x's words).
template <bool LSB, int NV>
__device__ __forceinline__ void gram_collect(u32 tmem, typename Gram<LSB, NV>::Shared& sh) {
    constexpr int V = 1 << NV;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const u32 addr = tmem + ((u32)(32 * (warp & 3)) << 16) + (warp >> 2) * 256;
    const int i = 2 * warp + (lane >> 4);
#pragma unroll 1
    for (int j = 0; j < V; j++) {
        const u64 v = tc_row_sum(addr + 16 * j, lane);
        if ((lane & 15) == 0) sh.g[V * i + j] = v;
    }
}

// Entry (p, p') of round k's two matrices from G; values are read at their
// place in the tables' groups (LSB: the index bits reversed).
template <bool LSB, int NV>
__device__ __forceinline__ void gram_round_matrices(typename Gram<LSB, NV>::Shared& sh) {
    constexpr int V = 1 << NV, NQ = Gram<LSB, NV>::NQ;
    for (int e = threadIdx.x; e < 2 * NQ; e += GR_TPB) {
        const int which = e >= NQ;
        int r = e - which * NQ, k = 0;
        while (r >= (1 << (2 * k))) { r -= 1 << (2 * k); k++; }
        const int p = r >> k, pp = r & ((1 << k) - 1);
        const int sb = NV - 1 - k;                     // suffix bits
        auto at = [&](int a, int b, int s) {
            u32 i = (p << (sb + 1)) | (a << sb) | s, j = (pp << (sb + 1)) | (b << sb) | s;
            if (LSB) { i = __brev(i) >> (32 - NV); j = __brev(j) >> (32 - NV); }
            return sh.g[V * i + j];
        };
        Acc pos = acc_zero(), neg = acc_zero();
        for (int s = 0; s < (1 << sb); s++) {
            acc_add64(pos, at(0, 0, s));
            if (which) {
                acc_add64(pos, at(1, 1, s));
                acc_add64(neg, at(0, 1, s));
                acc_add64(neg, at(1, 0, s));
            }
        }
        sh.q[which][e - which * NQ] = gl_sub(acc_reduce(pos), acc_reduce(neg));
    }
}

// Rounds 0 .. NV - 1, by warp 0: lane 8 which + p sums row p of the round's
// matrix against the weights and multiplies by w_p.
template <bool LSB, int NV>
__device__ __noinline__ void gram_rounds(typename Gram<LSB, NV>::Shared& sh, const RoundArgs& a) {
    const int lane = threadIdx.x & 31;
    WarpTx w = tx_load((const DevTranscript*)a.tx.tx, lane);
    const TxStream st = tx_stream(6, a.tx.hook, a.tx.hook_len, lane);
    if (lane < 3) sh.w[0][lane] = lane == 0 ? 1 : 0;
    __syncwarp();
    int off = 0;
#pragma unroll 1
    for (int k = 0; k < NV; k++) {
        const int n = 1 << k, which = lane >> 3, p = lane & 7;
        F3 wp = f3_zero();
        if (lane < 16 && p < n) {
            const u64* q = &sh.q[which][off + (p << k)];
            AccF<FOLD_FORM> c0, c1, c2;
            c0.zero(); c1.zero(); c2.zero();
            for (int j = 0; j < n; j++) {
                c0.mac(q[j], sh.w[j][0]);
                c1.mac(q[j], sh.w[j][1]);
                c2.mac(q[j], sh.w[j][2]);
            }
            wp = f3_make(sh.w[p][0], sh.w[p][1], sh.w[p][2]);
            const F3 v = f3_mul<true, true>(f3_make(c0.reduce(), c1.reduce(), c2.reduce()), wp);
            sh.v[which][p][0] = v.c0; sh.v[which][p][1] = v.c1; sh.v[which][p][2] = v.c2;
        }
        __syncwarp();
        u64 wire = 0;
        if (lane < 6) {
            Acc s = acc_zero();
            for (int j = 0; j < n; j++) acc_add64(s, sh.v[lane / 3][j][lane % 3]);
            wire = acc_reduce(s);
        }
        const u64 r = tx_step(w, st, 6, 3, wire, a.tx.hook, a.tx.hook_len, lane, sh.tot, sh.raw, sh.scr);
        if (lane < 6) a.tx.proof_wire[6 * k + lane] = wire;
        if (lane < 3) a.tx.proof_chal[3 * k + lane] = r;
        off += n * n;
        if (k + 1 < NV) {
            // w'_(p, 1) = w_p r, w'_(p, 0) = w_p - w_p r
            const F3 rr = f3_make(shfl64(r, 0), shfl64(r, 1), shfl64(r, 2));
            if (lane < n) {
                const F3 hi = f3_mul<true, true>(wp, rr), lo = f3_sub<true>(wp, hi);
                sh.w[2 * p][0] = lo.c0; sh.w[2 * p][1] = lo.c1; sh.w[2 * p][2] = lo.c2;
                sh.w[2 * p + 1][0] = hi.c0; sh.w[2 * p + 1][1] = hi.c1; sh.w[2 * p + 1][2] = hi.c2;
            }
            __syncwarp();
        }
    }
    tx_store((DevTranscript*)a.tx.tx, w, lane);
}

// MIRROR: the tables are in host memory; every word loaded is also written
// to the device buffers a.t[i].out[0] for the second pass.
// Block bid of nb takes the tiles bid, bid + nb, ...
template <bool LSB, int NV, bool MIRROR>
__device__ __forceinline__ void gram_body(const RoundArgs& a, u32 ntiles, u32 bid, u32 nb) {
    using GT = Gram<LSB, NV>;
    using Tile = TcTile<LSB, NV>;
    constexpr int S = GT::S, UPW = GT::UPW, AHEAD = GT::AHEAD, V = GT::V;
    constexpr u64 LIMIT = MIRROR ? GR_HOST_LIMIT_NS : GR_LIMIT_NS;
    extern __shared__ char gram_dyn[];
    __shared__ typename GT::Shared sh;
    char* stages = gram_dyn + ((1024 - (smem_u32(gram_dyn) & 1023)) & 1023);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        for (int s = 0; s < S; s++) {
            mbar_init(&sh.full[s], GR_LW);
            mbar_init(&sh.empty[s], 1);
        }
        mbar_init(&sh.done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int i = threadIdx.x; i < V * V; i += GR_TPB) sh.g[i] = 0;
    if (warp == GR_LW) tc_alloc(&sh.tmem, GT::COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const u32 tmem = sh.tmem;
    const u32 G = nb;
    const u32 mine = bid < ntiles ? (ntiles - 1 - bid) / G + 1 : 0;   // this block's tiles
    bool abort = false;
    if (warp < GR_LW) {
        const u64 N = a.L >> NV;
        const int t = Tile::table(warp * UPW);
        const u64* X = a.t[t].in[0];
        u64* M = MIRROR ? a.t[t].out[0] : nullptr;
        auto word = [&](u32 i, int u) {
            return Tile::word(warp * UPW + u, lane, (a.tile0 + bid + (u64)i * G) * 128, 64, N);
        };
        ulonglong2 v[AHEAD][UPW];
#pragma unroll
        for (int q = 0; q < AHEAD; q++)
            if ((u32)q < mine)
#pragma unroll
                for (int u = 0; u < UPW; u++) v[q][u] = __ldcs((const ulonglong2*)(X + word(q, u)));
        for (u32 i0 = 0; i0 < mine; i0 += AHEAD) {
#pragma unroll
            for (int q = 0; q < AHEAD; q++) {
                const u32 i = i0 + q;
                if (i >= mine) break;
                const u32 s = i % S, ph = (i / S) & 1u;
                abort |= !mbar_wait_step(&sh.empty[s], ph ^ 1u, a.no_wait | abort, LIMIT);
#pragma unroll
                for (int u = 0; u < UPW; u++) Tile::store(stages + s * Tile::BYTES, warp * UPW + u, lane, v[q][u]);
                if (MIRROR)
#pragma unroll
                    for (int u = 0; u < UPW; u++) *(ulonglong2*)(M + word(i, u)) = v[q][u];
                if (i + AHEAD < mine)
#pragma unroll
                    for (int u = 0; u < UPW; u++) v[q][u] = __ldcs((const ulonglong2*)(X + word(i + AHEAD, u)));
                if (lane == 0 && i + AHEAD + TC_PREFETCH < mine)
#pragma unroll
                    for (int u = 0; u < UPW; u++) l2_prefetch(X + word(i + AHEAD + TC_PREFETCH, u), 512);
                fence_async_shared();
                __syncwarp();
                if (lane == 0) mbar_arrive(&sh.full[s]);
            }
        }
    } else if (lane == 0) {
        for (u32 i = 0; i < mine; i++) {
            const u32 s = i % S, ph = (i / S) & 1u;
            if (!mbar_wait_bounded(&sh.full[s], ph, LIMIT)) { abort = true; break; }
            tc_fence_after();
            const u32 xb = smem_u32(stages) + s * Tile::BYTES, yb = xb + Tile::ATOMS * Tile::ATOM;
#pragma unroll
            for (int k = 0; k < 4; k++)        // 32 groups (rows) each
#pragma unroll
                for (int m = 0; m < Tile::ATOMS; m++)
                    tc_mma_f8(tmem + 256 * m, tc_desc(xb + m * Tile::ATOM + k * 4096, Tile::ATOM, 1024),
                              tc_desc(yb + k * 4096, Tile::ATOM, 1024), tc_idesc(128, 16 * V, true), i > 0 || k > 0);
            tc_commit(&sh.empty[s]);
        }
        tc_commit(&sh.done);     // also after an abort: every MMA issued so far
    }
    // the accumulators are final once `done` completes (the MMA thread's
    // commit covers everything it issued, an abort included)
    if (warp < GR_LW || lane == 0) {
        if (!mbar_wait_bounded(&sh.done, 0, 4 * LIMIT)) abort = true;
    }
    __syncwarp();
    tc_fence_after();
    const bool bad = __syncthreads_or(abort);
    if (!bad && mine && warp < 4 * Tile::ATOMS) gram_collect<LSB, NV>(tmem, sh);
    tc_fence_before();
    __syncthreads();
    if (warp == GR_LW) tc_dealloc(tmem, GT::COLS);
    if (bad) {
        if (threadIdx.x == 0 && a.status) *(volatile u32*)a.status = EFFSC_STATUS_TIMEOUT;
        return;
    }
    // the blocks' sums: the last block adds them up
    if (nb > 1) {
        for (int i = threadIdx.x; i < V * V; i += GR_TPB) a.partials[(u64)bid * V * V + i] = sh.g[i];
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) sh.last = atomicAdd(a.counter, 1u) == nb - 1;
        __syncthreads();
        if (!sh.last) return;
        __threadfence();
        if (threadIdx.x < 512) {
            constexpr u32 PARTS = 512 / (V * V);       // 8 (2) threads per entry
            const u32 g = threadIdx.x % (V * V), part = threadIdx.x / (V * V);
            Acc s = acc_zero();
#pragma unroll 16
            for (u32 b = part; b < nb; b += PARTS) acc_add64(s, __ldcg(&a.partials[(u64)b * V * V + g]));
            // (over more than two parts: summed in place, part by part)
            if (part < 2) sh.fin[part][g] = acc_reduce(s);
            __syncwarp();
            for (u32 p = 2; p < PARTS; p += 2) {
                asm volatile("bar.sync 1, 512;" ::: "memory");
                if (part == p || part == p + 1) sh.fin[part & 1][g] = gl_add(sh.fin[part & 1][g], acc_reduce(s));
            }
            asm volatile("bar.sync 1, 512;" ::: "memory");
            if (part == 0) sh.g[g] = gl_add(sh.fin[0][g], sh.fin[1][g]);
        }
        if (threadIdx.x == 0) *a.counter = 0;
        __syncthreads();
    }
    if (a.acc_mode != ACC_NONE) {
        // one chunk of the tables: carry G to the next chunk's launch
        for (int i = threadIdx.x; i < V * V; i += GR_TPB) {
            const u64 v = sh.g[i];
            if (a.acc_mode == ACC_FIRST) a.acc[i] = v;
            else if (a.acc_mode == ACC_MID) a.acc[i] = gl_add(a.acc[i], v);
            else sh.g[i] = gl_add(a.acc[i], v);
        }
        if (a.acc_mode != ACC_LAST) return;
        __syncthreads();
    }
    gram_round_matrices<LSB, NV>(sh);
    __syncthreads();
    if (warp == 0) gram_rounds<LSB, NV>(sh, a);
}

template <bool LSB, int NV, bool MIRROR>
__global__ void __launch_bounds__(GR_TPB, 1) k_ip_gram(RoundArgs a, u32 ntiles) {
    chain_enter();
    gram_body<LSB, NV, MIRROR>(a, ntiles, blockIdx.x, gridDim.x);
}
// The passes of many MSB proofs in one launch.
__global__ void __launch_bounds__(GR_TPB, 1) k_ip_gram_many(const TcSeg* segs, u32 nsegs, const RoundArgs* args) {
    __shared__ __align__(16) RoundArgs sa;
    const TcSeg sg = tc_segment(segs, nsegs, args, sa);
    gram_body<false, 4, false>(sa, sg.ntiles, blockIdx.x - sg.first_block, sg.nblocks);
}

u32 gram_max_tiles(void) { return GR_MAX_TILES; }
u32 tc_many_tiles(u64 total) {
    return (u32)tc_tiles_per_block(total, (u64)(max_grid() / 8), GR_MAX_TILES);
}

template <bool LSB, int NV, bool MIRROR>
static bool gram_inst(const RoundArgs& a, u32 ntiles, int grid, cudaStream_t s) {
    constexpr u32 SMEM = Gram<LSB, NV>::SMEM;
    static std::atomic<uint64_t> configured{0};
    if (!tc_allow_smem(k_ip_gram<LSB, NV, MIRROR>, SMEM, configured)) return false;
    return launch_chain(k_ip_gram<LSB, NV, MIRROR>, grid, GR_TPB, SMEM, s, a, ntiles);
}
bool launch_ip_gram_many(const TcSeg* segs, u32 nsegs, const RoundArgs* args, u32 grid, cudaStream_t s) {
    constexpr u32 SMEM = Gram<false, 4>::SMEM;
    static std::atomic<uint64_t> configured{0};
    if (!tc_allow_smem(k_ip_gram_many, SMEM, configured)) return false;
    k_ip_gram_many<<<grid, GR_TPB, SMEM, s>>>(segs, nsegs, args);
    return true;
}
bool launch_ip_gram(bool lsb, int nv, bool mirror, const RoundArgs& a, u32 ntiles, int grid, cudaStream_t s) {
    switch ((nv << 2) + (lsb ? 2 : 0) + (mirror ? 1 : 0)) {
    case 12: return gram_inst<false, 3, false>(a, ntiles, grid, s);
    case 13: return gram_inst<false, 3, true>(a, ntiles, grid, s);
    case 14: return gram_inst<true, 3, false>(a, ntiles, grid, s);
    case 15: return gram_inst<true, 3, true>(a, ntiles, grid, s);
    case 16: return gram_inst<false, 4, false>(a, ntiles, grid, s);
    case 17: return gram_inst<false, 4, true>(a, ntiles, grid, s);
    case 18: return gram_inst<true, 4, false>(a, ntiles, grid, s);
    case 19: return gram_inst<true, 4, true>(a, ntiles, grid, s);
    default: return false;
    }
}

}  // namespace effsc
