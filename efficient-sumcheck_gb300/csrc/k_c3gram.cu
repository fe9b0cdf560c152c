// k_c3gram.cu -- rounds 0 and 1 of a Coefficient proof with the degree-3
// product evaluator (coef01.cuh) on the tensor cores.
//
// The pass needs 15 sums of products P(y, x) = E F G of three bilinear forms
// of a quadruple (tables 0, 1, 2; F, G over Fp, E over Fp or Fp3).  F G is
// biquadratic, so its nine values on {0, 1, inf}^2 give it everywhere; E is
// bilinear, so its four entries do.  Every sum is therefore a combination with
// small integer coefficients of
//   sum over the quadruples of (entry of E) x (value of F G on the grid):
// a product of the 12 (4) words of E's quadruples with nine words each, the
// quadruples its inner dimension -- 4-bit digits on tcgen05 as in k_gram.cu
// (192 x 144, exact in f32 up to 2^16 quadruples a block).  The integer pipes
// keep ten differences and nine products with their reductions per quadruple
// where the points' form took 60 products, 15 reductions and ~100 adds.
//
// Measured, eq * f * g at n = 24 (table 0 in Fp3): 475 us on the integer pipes,
// 168 here (4.0 TB/s; HBM alone 99, ~20 the last block's sums and transcript
// steps).  Asking tiles into L2 ahead as k_gram.cu does made it 395 (24 to 56
// small requests per tile).
//
// One block per SM: three groups of four warps take turns at tiles of 128
// quadruples of tables 1 and 2 (a lane per quadruple), four warps load table
// 0, and one thread issues the MMAs.
#include "coef01.cuh"
#include "tc.cuh"

namespace effsc {

constexpr int CG_FGG = 3;                          // groups of four warps for F G
constexpr int CG_FGW = 4 * CG_FGG, CG_EW = 8;      // F G warps, table 0 warps
constexpr int CG_TPB = 32 * (CG_FGW + CG_EW + 1);
constexpr int CG_S = 3;                            // stages of 48 KB
static_assert(CG_S % CG_FGG == 0, "a stage is always filled by the same group: a barrier's phase parity tells its uses apart");
// A stage: words 0-7 of table 0, grid values 0-7, and a shared atom with grid
// value 8 in chunk 0 (the second operand's second atom) and words 8-11 in
// chunks 4-7 (the first operand's).  Three stages leave the loads in flight
// 100 KB of L1 (four atoms a stage left 60: 175 us against 168 at n = 24).
constexpr u32 CG_ATOM = 128 * 128, CG_BYTES = 3 * CG_ATOM;
constexpr u32 CG_SMEM = CG_S * CG_BYTES + 1024;
constexpr int CG_AHEAD = 2;                        // tiles of table 0 in registers
constexpr u64 CG_LIMIT_NS = 1000000000ULL;

struct C3Shared {
    u64 full[CG_S], empty[CG_S], done;
    u32 tmem;
    int last;
    u64 g[12 * 9];          // word 4 c + uv of table 0, grid value 3 y + x
    u64 fin[4][12 * 9];
    u64 part[C301_WORDS][4];
    u64 tot[C301_STRIDE];
};

// The row of a tile's quadruple q.  Eight lanes with eight neighbouring
// quadruples, or with every other one of sixteen, then store their chunks
// without bank conflicts.
__device__ __forceinline__ u32 c3_row(u32 q) { return q ^ ((q >> 3) & 1); }

// Table 0's 16-byte pieces: MSB, word w's quadruples 64 h + 2 lane and the
// next; LSB, entries (0, v), (1, v) of component c's quadruple 16 i + lane / 2,
// v = lane mod 2.
template <bool LSB, bool E0>
struct C3Units {
    static constexpr int NC = E0 ? 3 : 1, UNITS = 8 * NC, UPW = UNITS / CG_EW;
    __device__ __forceinline__ static const u64* at(const RoundArgs& a, int u, int lane, u64 k0, u64 Q) {
        if (LSB) return a.t[0].in[u >> 3] + 4 * (k0 + 16 * (u & 7) + (lane >> 1)) + 2 * (lane & 1);
        const int w = u >> 1;                      // 4 c + uv
        return a.t[0].in[w >> 2] + (w & 3) * Q + k0 + 64 * (u & 1) + 2 * lane;
    }
    // word w's chunk: atom 0 (w < 8) or chunk w - 4 of the shared one
    __device__ __forceinline__ static char* place(char* rows, u32 row, u32 w) {
        return rows + (w < 8 ? swz128(row, w) : 2 * CG_ATOM + swz128(row, w - 4));
    }
    __device__ __forceinline__ static void store(char* rows, int u, int lane, const ulonglong2& v) {
        if (LSB) {
            const u32 row = c3_row(16 * (u & 7) + (lane >> 1)), w = 4 * (u >> 3) + (lane & 1);
            *(uint4*)place(rows, row, w) = digits_of(v.x);
            *(uint4*)place(rows, row, w + 2) = digits_of(v.y);
        } else {
            const u32 w = u >> 1, q = 64 * (u & 1) + 2 * lane;
            *(uint4*)place(rows, c3_row(q), w) = digits_of(v.x);
            *(uint4*)place(rows, c3_row(q + 1), w) = digits_of(v.y);
        }
    }
};

// Quadruple k of tables 1 and 2, t_uv at 2 u + v.
template <bool LSB>
__device__ __forceinline__ void c3_load_fg(u64 (&t)[8], const RoundArgs& a, u64 k, u64 Q) {
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const u64* X = a.t[1 + i].in[0];
        if (LSB) {
            const ulonglong2 v0 = __ldcs((const ulonglong2*)(X + 4 * k)), v1 = __ldcs((const ulonglong2*)(X + 4 * k + 2));
            t[4 * i] = v0.x; t[4 * i + 2] = v0.y; t[4 * i + 1] = v1.x; t[4 * i + 3] = v1.y;
        } else {
#pragma unroll
            for (int j = 0; j < 4; j++) t[4 * i + j] = __ldcs(X + k + j * Q);
        }
    }
}
// A form's values at (y, x), 3 y + x over {0, 1, inf}^2.
__device__ __forceinline__ void c3_grid(u64 (&v)[9], const u64* t) {
    v[0] = t[0]; v[1] = t[1]; v[2] = gl_sub(t[1], t[0]);
    v[3] = t[2]; v[4] = t[3]; v[5] = gl_sub(t[3], t[2]);
    v[6] = gl_sub(t[2], t[0]); v[7] = gl_sub(t[3], t[1]); v[8] = gl_sub(v[5], v[2]);
}

// The 45 sums from the products: point i = 4 col + j (coef01.cuh) is E's form
// with weights (alpha_y, alpha_x) on its entries times F G's grid values with
// weights beta_y beta_x; y, x in 0, 1, 2, inf (3).
static __constant__ signed char c_c3_alpha[4][2] = {{1, 0}, {0, 1}, {-1, 2}, {-1, 1}};
static __constant__ signed char c_c3_beta[4][3] = {{1, 0, 0}, {0, 1, 0}, {-1, 2, 2}, {0, 0, 1}};
__device__ __forceinline__ void c3_sums(C3Shared& sh) {
    for (int e = threadIdx.x; e < C301_WORDS * 4; e += CG_TPB) {
        const int wd = e >> 2, uv = e & 3, i = wd / 3, c = wd - 3 * i, col = i >> 2, j = i & 3;
        const int x = col == 0 ? 0 : col == 1 ? 2 : col == 2 ? 3 : 1;
        const int y = col == 3 ? (j == 0 ? 0 : j + 1) : j;
        const int al = c_c3_alpha[y][uv >> 1] * c_c3_alpha[x][uv & 1];
        Acc pos = acc_zero(), neg = acc_zero();
#pragma unroll
        for (int g = 0; g < 9; g++) {
            const int k = al * c_c3_beta[y][g / 3] * c_c3_beta[x][g % 3];
            const u64 v = sh.g[(4 * c + uv) * 9 + g];
            if (k > 0) acc_mac(pos, v, (u64)k);
            if (k < 0) acc_mac(neg, v, (u64)-k);
        }
        sh.part[wd][uv] = gl_sub(acc_reduce(pos), acc_reduce(neg));
    }
    __syncthreads();
    if (threadIdx.x < C301_WORDS) {
        const u64* p = sh.part[threadIdx.x];
        sh.tot[threadIdx.x] = gl_add(gl_add(p[0], p[1]), gl_add(p[2], p[3]));
    }
}

template <bool LSB, bool E0>
__global__ void __launch_bounds__(CG_TPB, 1) k_c3_gram(RoundArgs a, u32 ntiles) {
    chain_enter();
    using U = C3Units<LSB, E0>;
    constexpr int BLOCKS = E0 ? 2 : 1, WORDS = 4 * U::NC;
    extern __shared__ char cg_dyn[];
    __shared__ C3Shared sh;
    char* stages = cg_dyn + ((1024 - (smem_u32(cg_dyn) & 1023)) & 1023);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        for (int s = 0; s < CG_S; s++) {
            mbar_init(&sh.full[s], 4 + CG_EW);
            mbar_init(&sh.empty[s], 1);
        }
        mbar_init(&sh.done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (threadIdx.x < 108) sh.g[threadIdx.x] = 0;
    if (warp == CG_FGW + CG_EW) tc_alloc(&sh.tmem, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const u32 tmem = sh.tmem;
    const u32 nb = gridDim.x;
    const u32 mine = blockIdx.x < ntiles ? (ntiles - 1 - blockIdx.x) / nb + 1 : 0;
    const u64 Q = a.L >> 2;
    auto tile_k0 = [&](u32 i) { return (a.tile0 + blockIdx.x + (u64)i * nb) * 128; };
    bool abort = false;
    if (warp < CG_FGW) {
        // a group's tiles are every CG_FGG-th; the next one's words are in flight
        const int group = warp >> 2, quad = 32 * (warp & 3) + lane;
        const u32 row = c3_row(quad);
        u64 t[8];
        if ((u32)group < mine) c3_load_fg<LSB>(t, a, tile_k0(group) + quad, Q);
        for (u32 i = group; i < mine; i += CG_FGG) {
            u64 f[9], g[9];
            c3_grid(f, t);
            c3_grid(g, t + 4);
#pragma unroll
            for (int q = 0; q < 9; q++) f[q] = gl_mul(f[q], g[q]);
            if (i + CG_FGG < mine) c3_load_fg<LSB>(t, a, tile_k0(i + CG_FGG) + quad, Q);
            const u32 s = i % CG_S;
            abort |= !mbar_wait_step(&sh.empty[s], ((i / CG_S) & 1u) ^ 1u, a.no_wait | abort);
            char* rows = stages + s * CG_BYTES + CG_ATOM;
#pragma unroll
            for (int q = 0; q < 9; q++)
                *(uint4*)(rows + (q >> 3) * CG_ATOM + swz128(row, q & 7)) = digits_of(f[q]);
            fence_async_shared();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.full[s]);
        }
    } else if (warp < CG_FGW + CG_EW) {
        const int w = warp - CG_FGW;
        ulonglong2 v[CG_AHEAD][U::UPW];
#pragma unroll
        for (int q = 0; q < CG_AHEAD; q++)
            if ((u32)q < mine)
#pragma unroll
                for (int u = 0; u < U::UPW; u++)
                    v[q][u] = __ldcs((const ulonglong2*)U::at(a, w * U::UPW + u, lane, tile_k0(q), Q));
        for (u32 i0 = 0; i0 < mine; i0 += CG_AHEAD) {
#pragma unroll
            for (int q = 0; q < CG_AHEAD; q++) {
                const u32 i = i0 + q;
                if (i >= mine) break;
                const u32 s = i % CG_S;
                abort |= !mbar_wait_step(&sh.empty[s], ((i / CG_S) & 1u) ^ 1u, a.no_wait | abort);
#pragma unroll
                for (int u = 0; u < U::UPW; u++) U::store(stages + s * CG_BYTES, w * U::UPW + u, lane, v[q][u]);
                if (i + CG_AHEAD < mine)
#pragma unroll
                    for (int u = 0; u < U::UPW; u++)
                        v[q][u] = __ldcs((const ulonglong2*)U::at(a, w * U::UPW + u, lane, tile_k0(i + CG_AHEAD), Q));
                fence_async_shared();
                __syncwarp();
                if (lane == 0) mbar_arrive(&sh.full[s]);
            }
        }
    } else if (lane == 0) {
        for (u32 i = 0; i < mine; i++) {
            const u32 s = i % CG_S;
            if (!mbar_wait_bounded(&sh.full[s], (i / CG_S) & 1u)) { abort = true; break; }
            tc_fence_after();
            const u32 xb = smem_u32(stages) + s * CG_BYTES, yb = xb + CG_ATOM;
#pragma unroll
            for (int k = 0; k < 4; k++)
#pragma unroll
                for (int m = 0; m < BLOCKS; m++)
                    tc_mma_f8(tmem + 256 * m, tc_desc(xb + 2 * m * CG_ATOM + k * 4096, CG_ATOM, 1024),
                              tc_desc(yb + k * 4096, CG_ATOM, 1024), tc_idesc(128, 144, true), i > 0 || k > 0);
            tc_commit(&sh.empty[s]);
        }
        tc_commit(&sh.done);
    }
    if (warp < CG_FGW + CG_EW || lane == 0) {
        if (!mbar_wait_bounded(&sh.done, 0, 4 * CG_LIMIT_NS)) abort = true;
    }
    __syncwarp();
    tc_fence_after();
    const bool bad = __syncthreads_or(abort);
    // words 0..7 in the first accumulator's 128 rows, 8..11 in the second's last 64
    if (!bad && mine && (warp < (E0 ? 4 : 2) || (E0 && (warp == 6 || warp == 7)))) {
        const u32 addr = tmem + ((u32)(32 * (warp & 3)) << 16) + (warp >> 2) * 256;
#pragma unroll 1
        for (int j = 0; j < 9; j++) {
            const u64 v = tc_row_sum(addr + 16 * j, lane);
            if ((lane & 15) == 0) sh.g[((warp < 4 ? 2 * warp : 2 * warp - 4) + (lane >> 4)) * 9 + j] = v;
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == CG_FGW + CG_EW) tc_dealloc(tmem, 512);
    if (bad) {
        if (threadIdx.x == 0 && a.status) *(volatile u32*)a.status = EFFSC_STATUS_TIMEOUT;
        return;
    }
    if (nb > 1) {
        if (threadIdx.x < 108) a.partials[(u64)blockIdx.x * 108 + threadIdx.x] = sh.g[threadIdx.x];
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) sh.last = atomicAdd(a.counter, 1u) == nb - 1;
        __syncthreads();
        if (!sh.last) return;
        __threadfence();
        if (threadIdx.x < 432) {
            const u32 g = threadIdx.x % 108, part = threadIdx.x / 108;
            Acc s = acc_zero();
#pragma unroll 8
            for (u32 b = part; b < nb; b += 4) acc_add64(s, __ldcg(&a.partials[(u64)b * 108 + g]));
            sh.fin[part][g] = acc_reduce(s);
        }
        __syncthreads();
        if (threadIdx.x < 108)
            sh.g[threadIdx.x] = gl_add(gl_add(sh.fin[0][threadIdx.x], sh.fin[1][threadIdx.x]),
                                       gl_add(sh.fin[2][threadIdx.x], sh.fin[3][threadIdx.x]));
        if (threadIdx.x == 0) *a.counter = 0;
        __syncthreads();
    }
    if (a.acc_mode != ACC_NONE) {
        // more quadruples than the accumulators hold: carry the sums to the next launch
        if (threadIdx.x < 108) {
            const u64 v = sh.g[threadIdx.x];
            if (a.acc_mode == ACC_FIRST) a.acc[threadIdx.x] = v;
            else if (a.acc_mode == ACC_MID) a.acc[threadIdx.x] = gl_add(a.acc[threadIdx.x], v);
            else sh.g[threadIdx.x] = gl_add(a.acc[threadIdx.x], v);
        }
        if (a.acc_mode != ACC_LAST) return;
        __syncthreads();
    }
    c3_sums(sh);
    __syncthreads();
    if (warp == 0) finalize_c301(sh.tot, a);
}

template <bool LSB, bool E0>
static bool c3_gram_inst(const RoundArgs& a, u32 ntiles, int grid, cudaStream_t s) {
    static std::atomic<uint64_t> configured{0};
    if (!tc_allow_smem(k_c3_gram<LSB, E0>, CG_SMEM, configured)) return false;
    return launch_chain(k_c3_gram<LSB, E0>, grid, CG_TPB, CG_SMEM, s, a, ntiles);
}
bool launch_c3_gram(bool lsb, bool e0, const RoundArgs& a, u32 ntiles, int grid, cudaStream_t s) {
    if (lsb) return e0 ? c3_gram_inst<true, true>(a, ntiles, grid, s) : c3_gram_inst<true, false>(a, ntiles, grid, s);
    return e0 ? c3_gram_inst<false, true>(a, ntiles, grid, s) : c3_gram_inst<false, false>(a, ntiles, grid, s);
}

}  // namespace effsc
