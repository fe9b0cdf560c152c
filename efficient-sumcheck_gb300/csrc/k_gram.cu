// k_gram.cu -- the first pass of the InnerProduct start (rounds 0-2) on the
// tensor cores.
//
// Every one of the pass's 26 sums (ip012.cuh) is a sum over the octets of
// (a linear form of x's eight values) times (the same form of y's), so all of
// them are linear in the 64 sums G_ij = sum_m x_i[m] y_j[m]: a Gram matrix, a
// matrix product with the octets as its inner dimension.  Split into 4-bit
// digits (tc.cuh) an octet of a table is 128 bytes, and G's digit sums are
// one 128 x 128 product over all octets, exact in f32 up to 74565 octets per
// accumulator.
//
// One block per SM.  Sixteen warps load the tables (each lane 16 bytes a
// time, GR_AHEAD tiles ahead, in registers), split the words and store the
// digit rows; a stage is GR_KT octets of both tables (row = octet, 128 bytes,
// 128-byte swizzle: the M / N index contiguous, as both operands of
// tcgen05.mma take it).  One thread of a seventeenth warp issues a stage's
// MMAs as soon as the stage is full and commits it empty.  At the end four
// warps read the 128 x 128 accumulators out of tensor memory and recombine
// the digits into 64 sums mod p; the last block to finish adds up the blocks'
// and derives the 26 sums for finalize_ip012.
//
// Measured (with the reduction and the three transcript steps, ~30 us): n = 26
// 310 -> 215 us (5.0 TB/s; 26 products per octet on the integer pipes before),
// LSB n = 24 121 -> 83 us; proofs 1132 -> 1038 and 498 -> 458 us.
// Bound: HBM (16 bytes per entry of the tables).  Per octet an SM spends
// about 1.8 cycles on the ALU (96 mask and shift instructions against the 530
// of 26 products with their differences), 4 on shared memory (256 bytes
// written, 256 read by the MMAs) and 2 on the tensor core, where the tables
// take 5.8 cycles to arrive.
#include "ip012.cuh"
#include "tc.cuh"

#include <atomic>

namespace effsc {

constexpr int GR_KT = 128;                    // octets per stage
constexpr int GR_S = 6;                       // stages of 32 KB
constexpr int GR_AHEAD = 4;                   // tiles in flight in registers
constexpr int GR_LW = 16;                     // loading warps
constexpr int GR_TPB = 32 * (GR_LW + 1);
constexpr u32 GR_HALF = GR_KT * 128;          // bytes of one table's rows
constexpr u32 GR_SMEM = GR_S * 2 * GR_HALF + 1024;
constexpr u32 GR_MAX_TILES = 65536 / GR_KT;   // tiles per accumulator: 2^16 octets (2^16 * 225 < 2^24)
constexpr u64 GR_LIMIT_NS = 1000000000ULL;

// The sums' forms: values added and subtracted (bit i: value i = 4 t0 + 2 t1 + t2).
static __constant__ unsigned char c_form_pos[IP012_WORDS] = {
    0x01, 0x04, 0x04, 0x10, 0x40, 0x40, 0x10, 0x40, 0x41, 0x02, 0x20, 0x20, 0x08, 0x80,
    0x02, 0x08, 0x09, 0x20, 0x80, 0x90, 0x21, 0x84, 0x96, 0x08, 0x80, 0x82};
static __constant__ unsigned char c_form_neg[IP012_WORDS] = {
    0x00, 0x00, 0x01, 0x00, 0x00, 0x10, 0x01, 0x04, 0x14, 0x00, 0x00, 0x02, 0x00, 0x08,
    0x01, 0x04, 0x06, 0x10, 0x40, 0x60, 0x12, 0x48, 0x69, 0x02, 0x20, 0x28};

struct GramShared {
    u64 full[GR_S], empty[GR_S], done;
    u32 tmem;
    int abort, last;
    u64 g[64];
    u64 fin[8][64];
    u64 rows[IP012_WORDS][8];
    u64 tot[32];
};

// The two 16-byte pieces a lane loads of a tile: MSB, slice j = w of the
// warp's table, octets 64 h + 2 lane and the next (kept in rows 64 h + lane
// and 64 h + 32 + lane: the order of the octets within a tile is free, and
// this one stores without bank conflicts); LSB, entries 2 q, 2 q + 1 of octet
// 16 w + 8 h + lane / 4, q = lane mod 4.
template <bool LSB>
__device__ __forceinline__ u64 gram_word(u64 tile, int w, int h, int lane, u64 O) {
    if (LSB) return (tile * GR_KT + 16 * w + 8 * h + (lane >> 2)) * 8 + 2 * (lane & 3);
    return (u64)w * O + tile * GR_KT + 64 * h + 2 * lane;
}
template <bool LSB>
__device__ __forceinline__ void gram_store(char* rows, int w, int h, int lane, const ulonglong2& v) {
    if (LSB) {
        const u32 row = 16 * w + 8 * h + (lane >> 2), q = 2 * (lane & 3);
        *(uint4*)(rows + swz128(row, q)) = digits_of(v.x);
        *(uint4*)(rows + swz128(row, q + 1)) = digits_of(v.y);
    } else {
        const u32 row = 64 * h + lane;
        *(uint4*)(rows + swz128(row, w)) = digits_of(v.x);
        *(uint4*)(rows + swz128(row + 32, w)) = digits_of(v.y);
    }
}

// Digit sums of four warps' accumulator rows -> G (added to sh.g).  Row
// 32 warp + lane is digit d = row mod 16 of x's value row / 16.
__device__ __forceinline__ void gram_collect(u32 tmem, GramShared& sh) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const u32 d = lane & 15, sft = 4 * (d < 8 ? 2 * d : 2 * (d - 8) + 1);   // this row's weight 2^sft
#pragma unroll 1
    for (int j = 0; j < 8; j++) {
        float f[16];
        tc_ld16(f, tmem + ((u32)(32 * warp) << 16) + 16 * j);
        tc_wait_ld();
        u64 lo = 0, hi = 0;
#pragma unroll
        for (int b = 7; b >= 0; b--) {
            // low and high digit of byte b: below 2^29
            const u32 s = (u32)(f[b] * 262144.0f) + 16 * (u32)(f[8 + b] * 262144.0f);
            if (b >= 4) hi = (hi << 8) + s;
            else lo = (lo << 8) + s;
        }
        // lo + hi 2^32, below 2^86
        const u64 mid = (lo >> 32) + (hi & 0xFFFFFFFFu);
        u64 v = gl_reduce_limbs((u32)lo, (u32)mid, (u32)((hi >> 32) + (mid >> 32)), 0, 0);
        v = gl_mul(v, 1ULL << sft);
#pragma unroll
        for (int o = 8; o; o >>= 1) v = gl_add(v, __shfl_xor_sync(0xffffffffu, v, o));
        if (d == 0) {
            u64& g = sh.g[8 * (2 * warp + (lane >> 4)) + j];
            g = gl_add(g, v);
        }
    }
}

// MIRROR: the tables are in host memory; every word loaded is also written
// to the device buffers a.t[i].out[0] for the second pass.
template <bool LSB, bool MIRROR>
__global__ void __launch_bounds__(GR_TPB, 1) k_ip_gram(RoundArgs a, u32 ntiles) {
    chain_enter();
    extern __shared__ char gram_dyn[];
    __shared__ GramShared sh;
    char* stages = gram_dyn + ((1024 - (smem_u32(gram_dyn) & 1023)) & 1023);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        for (int s = 0; s < GR_S; s++) {
            mbar_init(&sh.full[s], GR_LW);
            mbar_init(&sh.empty[s], 1);
        }
        mbar_init(&sh.done, 1);
        sh.abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (threadIdx.x < 64) sh.g[threadIdx.x] = 0;
    if (warp == GR_LW) tc_alloc(&sh.tmem, 128);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const u32 tmem = sh.tmem;
    const u32 G = gridDim.x;
    const u32 mine = blockIdx.x < ntiles ? (ntiles - 1 - blockIdx.x) / G + 1 : 0;   // this block's tiles
    bool abort = false;
    if (warp < GR_LW) {
        const u64 O = a.L >> 3;
        const int t = warp >> 3, w = warp & 7;
        const u64* X = a.t[t].in[0];
        u64* M = MIRROR ? a.t[t].out[0] : nullptr;
        char* rows = stages + t * GR_HALF;
        ulonglong2 v[GR_AHEAD][2];
#pragma unroll
        for (int q = 0; q < GR_AHEAD; q++)
            if ((u32)q < mine)
#pragma unroll
                for (int h = 0; h < 2; h++)
                    v[q][h] = *(const ulonglong2*)(X + gram_word<LSB>(a.tile0 + blockIdx.x + (u64)q * G, w, h, lane, O));
        for (u32 i0 = 0; i0 < mine && !abort; i0 += GR_AHEAD) {
#pragma unroll
            for (int q = 0; q < GR_AHEAD; q++) {
                const u32 i = i0 + q;
                if (i >= mine || abort) break;
                const u32 s = i % GR_S, ph = (i / GR_S) & 1u;
                if (!mbar_wait_bounded(&sh.empty[s], ph ^ 1u)) { abort = true; break; }
#pragma unroll
                for (int h = 0; h < 2; h++) gram_store<LSB>(rows + s * 2 * GR_HALF, w, h, lane, v[q][h]);
                if (MIRROR)
#pragma unroll
                    for (int h = 0; h < 2; h++)
                        *(ulonglong2*)(M + gram_word<LSB>(a.tile0 + blockIdx.x + (u64)i * G, w, h, lane, O)) = v[q][h];
                if (i + GR_AHEAD < mine)
#pragma unroll
                    for (int h = 0; h < 2; h++)
                        v[q][h] = *(const ulonglong2*)(X + gram_word<LSB>(a.tile0 + blockIdx.x + (u64)(i + GR_AHEAD) * G, w, h, lane, O));
                fence_async_shared();
                __syncwarp();
                if (lane == 0) mbar_arrive(&sh.full[s]);
            }
        }
    } else if (lane == 0) {
        for (u32 i = 0; i < mine; i++) {
            const u32 s = i % GR_S, ph = (i / GR_S) & 1u;
            if (!mbar_wait_bounded(&sh.full[s], ph)) { abort = true; break; }
            tc_fence_after();
            const u32 base = smem_u32(stages) + s * 2 * GR_HALF;
#pragma unroll
            for (int k = 0; k < GR_KT / 32; k++)
                tc_mma_f8(tmem, tc_desc(base + k * 4096, 1024), tc_desc(base + GR_HALF + k * 4096, 1024),
                          tc_idesc(128, 128, true), i > 0 || k > 0);
            tc_commit(&sh.empty[s]);
        }
        tc_commit(&sh.done);     // also after an abort: every MMA issued so far
    }
    // the accumulators are final once `done` completes (the MMA thread's
    // commit covers everything it issued, an abort included)
    if (warp < GR_LW || lane == 0) {
        if (!mbar_wait_bounded(&sh.done, 0, 4 * GR_LIMIT_NS)) abort = true;
    }
    __syncwarp();
    tc_fence_after();
    const bool bad = __syncthreads_or(abort);
    if (!bad && mine && warp < 4) gram_collect(tmem, sh);
    tc_fence_before();
    __syncthreads();
    if (warp == GR_LW) tc_dealloc(tmem, 128);
    if (bad) {
        if (threadIdx.x == 0 && a.status) *(volatile u32*)a.status = EFFSC_STATUS_TIMEOUT;
        return;
    }
    // the blocks' sums: the last block adds them up
    const u32 nb = gridDim.x;
    if (nb > 1) {
        if (threadIdx.x < 64) a.partials[(u64)blockIdx.x * 64 + threadIdx.x] = sh.g[threadIdx.x];
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) sh.last = atomicAdd(a.counter, 1u) == nb - 1;
        __syncthreads();
        if (!sh.last) return;
        __threadfence();
        if (threadIdx.x < 512) {
            const u32 g = threadIdx.x & 63, part = threadIdx.x >> 6;
            Acc s = acc_zero();
#pragma unroll 4
            for (u32 b = part; b < nb; b += 8) acc_add64(s, __ldcg(&a.partials[(u64)b * 64 + g]));
            sh.fin[part][g] = acc_reduce(s);
        }
        __syncthreads();
        if (threadIdx.x < 64) {
            Acc s = acc_zero();
#pragma unroll
            for (int p = 0; p < 8; p++) acc_add64(s, sh.fin[p][threadIdx.x]);
            sh.g[threadIdx.x] = acc_reduce(s);
        }
        if (threadIdx.x == 0) *a.counter = 0;
        __syncthreads();
    }
    // sum s = (form s of x) (form s of y): over y's values for each of x's, then over x's
    if (threadIdx.x < IP012_WORDS * 8) {
        const int s = threadIdx.x >> 3, i = threadIdx.x & 7;
        const u32 pos = c_form_pos[s], neg = c_form_neg[s];
        const int ri = LSB ? ((i & 1) << 2) | (i & 2) | (i >> 2) : i;
        Acc p = acc_zero(), n = acc_zero();
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const int rj = LSB ? ((j & 1) << 2) | (j & 2) | (j >> 2) : j;
            const u64 g = sh.g[8 * ri + rj];
            if ((pos >> j) & 1u) acc_add64(p, g);
            if ((neg >> j) & 1u) acc_add64(n, g);
        }
        sh.rows[s][i] = gl_sub(acc_reduce(p), acc_reduce(n));
    }
    __syncthreads();
    if (threadIdx.x < IP012_WORDS) {
        const u32 pos = c_form_pos[threadIdx.x], neg = c_form_neg[threadIdx.x];
        Acc p = acc_zero(), n = acc_zero();
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const u64 r = sh.rows[threadIdx.x][i];
            if ((pos >> i) & 1u) acc_add64(p, r);
            if ((neg >> i) & 1u) acc_add64(n, r);
        }
        sh.tot[threadIdx.x] = gl_sub(acc_reduce(p), acc_reduce(n));
    }
    __syncthreads();
    if (a.acc_mode != ACC_NONE) {
        // one chunk of the tables: carry the sums to the next chunk's launch
        if (threadIdx.x < IP012_WORDS) {
            const u64 v = sh.tot[threadIdx.x];
            if (a.acc_mode == ACC_FIRST) a.acc[threadIdx.x] = v;
            else if (a.acc_mode == ACC_MID) a.acc[threadIdx.x] = gl_add(a.acc[threadIdx.x], v);
            else sh.tot[threadIdx.x] = gl_add(a.acc[threadIdx.x], v);
        }
        if (a.acc_mode != ACC_LAST) return;
        __syncthreads();
    }
    if (warp == 0) finalize_ip012(sh.tot, a);
}

u32 gram_tile_octets(void) { return GR_KT; }
u32 gram_max_tiles(void) { return GR_MAX_TILES; }

template <bool LSB, bool MIRROR>
static bool gram_inst(const RoundArgs& a, u32 ntiles, int grid, cudaStream_t s) {
    static std::atomic<uint64_t> configured{0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    const uint64_t bit = 1ull << (dev & 63);
    if (!(configured.load() & bit)) {
        if (cudaFuncSetAttribute(k_ip_gram<LSB, MIRROR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GR_SMEM) != cudaSuccess)
            return false;
        configured.fetch_or(bit);
    }
    return launch_chain(k_ip_gram<LSB, MIRROR>, grid, GR_TPB, GR_SMEM, s, a, ntiles);
}
bool launch_ip_gram(bool lsb, bool mirror, const RoundArgs& a, u32 ntiles, int grid, cudaStream_t s) {
    if (lsb) return mirror ? gram_inst<true, true>(a, ntiles, grid, s) : gram_inst<true, false>(a, ntiles, grid, s);
    return mirror ? gram_inst<false, true>(a, ntiles, grid, s) : gram_inst<false, false>(a, ntiles, grid, s);
}

}  // namespace effsc
