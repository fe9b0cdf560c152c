// k_tcfold.cu -- the second pass of the InnerProduct start on the tensor
// cores: fold both base tables with r_0 .. r_{NV-1} at once, write the Fp3
// tables of length L / 2^NV and evaluate round NV on them.
//
// An entry of the folded table is sum_v E_v x_v over its item's 2^NV words,
// E_v = prod_i (t_i ? r_i : 1 - r_i) (src/inner_product_sumcheck.rs:143-176
// applied NV times).  With x_v = sum_e digit_e 16^w(e) that is a matrix
// product: the digit rows of the tables (tc.cuh; 128 items to a tile, the
// digits contiguous: K) times a constant matrix of 48 columns, column
// 16 c + d the 4-bit digit d of component c of E_v 16^w(e) mod p.  Sums stay
// at most 256 * 225 < 2^16, exact in f32.  What is left for the integer pipes is
// to put sixteen digit sums back together per component (two per
// multiply-add in float, then four 32-bit pieces per 64-bit sum) instead of
// 3 (2^NV - 1) products with their differences per entry.
//
// One block per SM: sixteen loading warps as in the first pass (k_gram.cu),
// one warp whose first lane issues the MMAs, and two groups of four warps
// that take turns reading a tile's sums out of tensor memory (a lane per
// item, both tables), write the entries and accumulate the round's products:
// a folded pair's two halves sit in two lanes of a warp, the low half's lane
// sums a_lo b_lo and the high half's (a_hi - a_lo)(b_hi - b_lo), one product
// each.
//
// Measured, n = 26: the triple fold and round 3 on the integer pipes 373 us
// (and round 4 another 120); the fourfold fold and round 4 here 280 us
// with three stages, 245 (5.2 TB/s) with two: the loads in flight need the L1
// that the stages leave (asking tiles into L2 ahead, 268, then costs more than it
// gives).  Not faster: a third group of epilogue warps (284 against 274 us, at
// fewer registers), a third tile in registers (spills, 356), tensor-memory
// loads one component ahead, streaming stores.
#include "tc.cuh"

namespace effsc {

constexpr int TF_LW = 16;                     // loading warps
constexpr int TF_EG = 2;                      // groups of four epilogue warps
constexpr int TF_TPB = 32 * (TF_LW + 4 * TF_EG + 1);
constexpr int TF_MMA = TF_LW + 4 * TF_EG;     // the issuing warp
constexpr int TF_BUFS = 4;                    // accumulators in tensor memory, 128 columns each

template <bool LSB, int NV>
struct TcFold {
    using Tile = TcTile<LSB, NV>;
    static constexpr int V = 1 << NV;
    static constexpr int UPW = Tile::UNITS / TF_LW;
    static constexpr int AHEAD = NV == 3 ? 4 : 2;
    static constexpr u32 WBYTES = 48 * 128 * Tile::ATOMS;
    static constexpr int S = NV == 3 ? 4 : 2;      // stages: the rest is L1 for the loads in flight
    static constexpr u32 SMEM = S * Tile::BYTES + WBYTES + 1024;
    struct Shared {
        u64 full[S], empty[S], tfull[TF_BUFS], tempty[TF_BUFS], done;
        u32 tmem;
        int last;
        u64 e[V][3];
        u64 red[4 * TF_EG][2][3];
        u64 tot[12];
    };
};

// c0 + c1 2^32 + c2 2^64 mod p, canonical: u = (c1:c0) + c2 (2^32 - 1); a carry
// out is worth 2^32 - 1 once more and cannot carry again.
__device__ __forceinline__ u64 reduce96(u32 c0, u32 c1, u32 c2) {
    u32 r0, r1;
    asm("{\n\t.reg .u32 u0, u1, k, v0, v1, ge;\n\t.reg .pred q;\n\t"
        "mad.lo.cc.u32 u0, %4, 0xFFFFFFFF, %2;\n\t"
        "madc.hi.cc.u32 u1, %4, 0xFFFFFFFF, %3;\n\t"
        "addc.u32 k, 0, 0;\n\t"
        "neg.s32 k, k;\n\t"
        "add.cc.u32 u0, u0, k;\n\t"
        "addc.u32 u1, u1, 0;\n\t"
        "add.cc.u32 v0, u0, 0xFFFFFFFF;\n\t"
        "addc.cc.u32 v1, u1, 0;\n\t"
        "addc.u32 ge, 0, 0;\n\t"
        "setp.ne.u32 q, ge, 0;\n\t"
        "selp.b32 %0, v0, u0, q;\n\t"
        "selp.b32 %1, v1, u1, q;\n\t}"
        : "=r"(r0), "=r"(r1) : "r"(c0), "r"(c1), "r"(c2));
    return mk64(r0, r1);
}
// sum_d s_d 16^d mod p from sixteen sums below 2^16 given as s_d 2^-18.
__device__ __forceinline__ u64 join_digits(const float (&f)[16]) {
    // s_2i + 16 s_(2i+1) < 2^21 in the low bits of 2^23 + it
    u32 b[8];
#pragma unroll
    for (int i = 0; i < 8; i++)
        b[i] = __float_as_uint(__fmaf_rn(f[2 * i + 1], 16.0f * 262144.0f, __fmaf_rn(f[2 * i], 262144.0f, 8388608.0f)));
    constexpr u64 BIAS = 0ULL - 0x4B000000ULL * 0x01010101ULL;    // the four pieces' exponent bits come off
    u64 lo = BIAS + b[0], hi = BIAS + b[4];
#pragma unroll
    for (int i = 1; i < 4; i++) {
        lo += (u64)b[i] * (1u << (8 * i));
        hi += (u64)b[4 + i] * (1u << (8 * i));
    }
    // lo + hi 2^32 < 2^78
    u32 c1, c2;
    asm("add.cc.u32 %0, %2, %3;\n\taddc.u32 %1, %4, 0;" : "=r"(c1), "=r"(c2) : "r"(hi32(lo)), "r"(lo32(hi)), "r"(hi32(hi)));
    return reduce96(lo32(lo), c1, c2);
}

// Block bid of nb takes the tiles bid, bid + nb, ...
template <bool LSB, int NV>
__device__ __forceinline__ void tc_fold_body(const RoundArgs& a, u32 ntiles, u32 bid, u32 nb) {
    using FT = TcFold<LSB, NV>;
    using Tile = TcTile<LSB, NV>;
    constexpr int S = FT::S, UPW = FT::UPW, AHEAD = FT::AHEAD, V = FT::V;
    extern __shared__ char tf_dyn[];
    __shared__ typename FT::Shared sh;
    char* stages = tf_dyn + ((1024 - (smem_u32(tf_dyn) & 1023)) & 1023);
    char* wmat = stages + S * Tile::BYTES;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        for (int s = 0; s < S; s++) {
            mbar_init(&sh.full[s], TF_LW);
            mbar_init(&sh.empty[s], 1);
        }
        for (int s = 0; s < TF_BUFS; s++) {
            mbar_init(&sh.tfull[s], 1);
            mbar_init(&sh.tempty[s], 4);
        }
        mbar_init(&sh.done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == TF_MMA) tc_alloc(&sh.tmem, 128 * TF_BUFS);
    // E_v at the value's place in a group (LSB: index bits reversed)
    if (threadIdx.x < V) {
        F3 e = f3_make(1, 0, 0);
        for (int i = 0; i < NV; i++) {
            const F3 r = f3_make(a.chal_ptr[3 * i], a.chal_ptr[3 * i + 1], a.chal_ptr[3 * i + 2]);
            const F3 er = f3_mul<true, true>(e, r);
            const bool bit = LSB ? (threadIdx.x >> i) & 1 : (threadIdx.x >> (NV - 1 - i)) & 1;
            e = bit ? er : f3_sub<true>(e, er);
        }
        sh.e[threadIdx.x][0] = e.c0; sh.e[threadIdx.x][1] = e.c1; sh.e[threadIdx.x][2] = e.c2;
    }
    __syncthreads();
    // the constant matrix: row (column of the product) 16 c + d, byte 16 v + e
    for (int i = threadIdx.x; i < 3 * 16 * V; i += TF_TPB) {
        const int c = i / (16 * V), k = i % (16 * V), d = k & 15;
        const u64 m = gl_mul(sh.e[k >> 4][c], 1ULL << (4 * (d < 8 ? 2 * d : 2 * (d - 8) + 1)));
        char* col = wmat + (k >> 7) * (48 * 128);
        for (int q = 0; q < 16; q++)
            col[swz128(16 * c + q, (k & 127) >> 4) + (k & 15)] = (char)((m >> (4 * q)) & 15);
    }
    fence_async_shared();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const u32 tmem = sh.tmem;
    const u32 G = nb;
    const u32 mine = bid < ntiles ? (ntiles - 1 - bid) / G + 1 : 0;
    const u64 N = a.L >> NV, H = N >> 1;
    bool abort = false;
    ProdAcc<true, true> acc;
    acc.init();
    if (warp < TF_LW) {
        const int t = Tile::table(warp * UPW);
        const u64* X = a.t[t].in[0];
        auto word = [&](u32 i, int u) {
            const u64 tile = bid + (u64)i * G;
            return Tile::word(warp * UPW + u, lane, tile * (LSB ? 128 : 64), H, N);
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
                abort |= !mbar_wait_step(&sh.empty[s], ph ^ 1u, a.no_wait | abort);
#pragma unroll
                for (int u = 0; u < UPW; u++) Tile::store(stages + s * Tile::BYTES, warp * UPW + u, lane, v[q][u]);
                if (i + AHEAD < mine)
#pragma unroll
                    for (int u = 0; u < UPW; u++) v[q][u] = __ldcs((const ulonglong2*)(X + word(i + AHEAD, u)));
                fence_async_shared();
                __syncwarp();
                if (lane == 0) mbar_arrive(&sh.full[s]);
            }
        }
    } else if (warp == TF_MMA) {
        if (lane == 0) {
            const u32 wb = smem_u32(wmat);
            for (u32 i = 0; i < mine; i++) {
                const u32 s = i % S, b = i % TF_BUFS;
                if (!mbar_wait_bounded(&sh.full[s], (i / S) & 1u) ||
                    !mbar_wait_bounded(&sh.tempty[b], ((i / TF_BUFS) & 1u) ^ 1u)) { abort = true; break; }
                tc_fence_after();
                const u32 base = smem_u32(stages) + s * Tile::BYTES;
#pragma unroll
                for (int t = 0; t < 2; t++)
#pragma unroll
                    for (int k = 0; k < 4 * Tile::ATOMS; k++) {
                        const u32 at = k >> 2, in = (k & 3) * 32;       // atom, bytes into its rows
                        tc_mma_f8(tmem + 128 * b + 64 * t, tc_desc(base + (t * Tile::ATOMS + at) * Tile::ATOM + in, 1024, 1024),
                                  tc_desc(wb + at * (48 * 128) + in, 1024, 1024), tc_idesc(128, 48, false), k > 0);
                    }
                tc_commit(&sh.empty[s]);
                tc_commit(&sh.tfull[b]);
            }
            // no MMA is in flight when tensor memory is given back, an abort included
            tc_commit(&sh.done);
            if (!mbar_wait_bounded(&sh.done, 0)) abort = true;
        }
        __syncwarp();
    } else {
        const int e = warp - TF_LW, group = e >> 2, quad = warp & 3;
        const u32 addr = tmem + ((u32)(32 * quad) << 16);
        const bool high = lane >= 16;
        for (u32 i = group; i < mine; i += TF_EG) {
            const u32 b = i % TF_BUFS;
            abort |= !mbar_wait_step(&sh.tfull[b], (i / TF_BUFS) & 1u, a.no_wait | abort);
            __syncwarp();          // the loads are instructions of the whole warp
            tc_fence_after();
            const u64 m = Tile::entry(quad, lane, (bid + (u64)i * G) * (LSB ? 128 : 64), H);
            F3 x[2];
#pragma unroll
            for (int t = 0; t < 2; t++) {
                float f[16];
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    tc_ld16(f, addr + 128 * b + 64 * t + 16 * c);
                    tc_wait_ld(f);
                    if (t == 1 && c == 2) {
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&sh.tempty[b]);
                    }
                    const u64 w = join_digits(f);
                    a.t[t].out[c][m] = w;
                    if (c == 0) x[t].c0 = w;
                    if (c == 1) x[t].c1 = w;
                    if (c == 2) x[t].c2 = w;
                }
            }
            // the high half's lane takes the differences to its partner
#pragma unroll
            for (int t = 0; t < 2; t++) {
                const u64 p0 = __shfl_xor_sync(0xffffffffu, x[t].c0, Tile::PARTNER), p1 = __shfl_xor_sync(0xffffffffu, x[t].c1, Tile::PARTNER),
                          p2 = __shfl_xor_sync(0xffffffffu, x[t].c2, Tile::PARTNER);
                x[t] = f3_sub<true>(x[t], f3_make(high ? p0 : 0, high ? p1 : 0, high ? p2 : 0));
            }
            acc.mac(x[0], x[1]);
        }
        // q0 over the low halves' lanes, qinf over the high ones'
        F3 r = acc.result();
#pragma unroll
        for (int o = 8; o; o >>= 1) {
            r.c0 = gl_add(r.c0, __shfl_xor_sync(0xffffffffu, r.c0, o));
            r.c1 = gl_add(r.c1, __shfl_xor_sync(0xffffffffu, r.c1, o));
            r.c2 = gl_add(r.c2, __shfl_xor_sync(0xffffffffu, r.c2, o));
        }
        if ((lane & 15) == 0) {
            u64* d = sh.red[e][lane >> 4];
            d[0] = r.c0; d[1] = r.c1; d[2] = r.c2;
        }
    }
    tc_fence_before();
    const bool bad = __syncthreads_or(abort);
    tc_fence_after();
    if (warp == TF_MMA) tc_dealloc(tmem, 128 * TF_BUFS);
    if (bad) {
        if (threadIdx.x == 0 && a.status) *(volatile u32*)a.status = EFFSC_STATUS_TIMEOUT;
        return;
    }
    if (threadIdx.x < 6) {
        u64 s = 0;
#pragma unroll
        for (int w = 0; w < 4 * TF_EG; w++) s = gl_add(s, (&sh.red[w][0][0])[threadIdx.x]);
        if (nb == 1) sh.tot[threadIdx.x] = s;
        else a.partials[(u64)bid * 6 + threadIdx.x] = s;
    }
    if (nb > 1) {
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) sh.last = atomicAdd(a.counter, 1u) == nb - 1;
        __syncthreads();
        if (!sh.last) return;
        __threadfence();
        // warp w < 6 sums word w
        if (warp < 6) {
            Acc s = acc_zero();
#pragma unroll 8
            for (u32 b = lane; b < nb; b += 32) acc_add64(s, __ldcg(&a.partials[(u64)b * 6 + warp]));
            u64 v = acc_reduce(s);
#pragma unroll
            for (int o = 16; o; o >>= 1) v = gl_add(v, __shfl_xor_sync(0xffffffffu, v, o));
            if (lane == 0) sh.tot[warp] = v;
        }
        if (threadIdx.x == 0) *a.counter = 0;
    }
    if (threadIdx.x >= 6 && threadIdx.x < 12) sh.tot[threadIdx.x] = 0;
    __syncthreads();
    if (warp == 0) finalize_warp(POL_IP, sh.tot, a);
}

template <bool LSB, int NV>
__global__ void __launch_bounds__(TF_TPB, 1) k_tc_fold(RoundArgs a, u32 ntiles) {
    chain_enter();
    tc_fold_body<LSB, NV>(a, ntiles, blockIdx.x, gridDim.x);
}
// The passes of many MSB proofs in one launch.
__global__ void __launch_bounds__(TF_TPB, 1) k_tc_fold_many(const TcSeg* segs, u32 nsegs, const RoundArgs* args) {
    __shared__ __align__(16) RoundArgs sa;
    const TcSeg sg = tc_segment(segs, nsegs, args, sa);
    tc_fold_body<false, 4>(sa, sg.ntiles, blockIdx.x - sg.first_block, sg.nblocks);
}

template <bool LSB, int NV>
static bool fold_inst(bool copied, const RoundArgs& a, u32 ntiles, int grid, cudaStream_t s) {
    constexpr u32 SMEM = TcFold<LSB, NV>::SMEM;
    static std::atomic<uint64_t> configured{0};
    if (!tc_allow_smem(k_tc_fold<LSB, NV>, SMEM, configured)) return false;
    return launch_with(pdl_on(false) && !copied, k_tc_fold<LSB, NV>, grid, TF_TPB, SMEM, s, a, ntiles);
}
bool launch_tc_fold_many(const TcSeg* segs, u32 nsegs, const RoundArgs* args, u32 grid, cudaStream_t s) {
    constexpr u32 SMEM = TcFold<false, 4>::SMEM;
    static std::atomic<uint64_t> configured{0};
    if (!tc_allow_smem(k_tc_fold_many, SMEM, configured)) return false;
    k_tc_fold_many<<<grid, TF_TPB, SMEM, s>>>(segs, nsegs, args);
    return true;
}
bool launch_tc_fold(bool lsb, int nv, bool copied, const RoundArgs& a, u32 ntiles, int grid, cudaStream_t s) {
    if (nv == 3) return lsb ? fold_inst<true, 3>(copied, a, ntiles, grid, s) : fold_inst<false, 3>(copied, a, ntiles, grid, s);
    if (nv == 4) return lsb ? fold_inst<true, 4>(copied, a, ntiles, grid, s) : fold_inst<false, 4>(copied, a, ntiles, grid, s);
    return false;
}

}  // namespace effsc
