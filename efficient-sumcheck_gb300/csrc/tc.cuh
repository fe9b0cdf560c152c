// tc.cuh -- what the tensor-core passes share: tcgen05 instructions, operand
// descriptors, and exact integer products from 8-bit floats.
//
// A 64-bit word is sixteen 4-bit digits.  As the low bits of an e4m3 byte a
// digit n in 0..15 is the number n 2^-9 (0..7 subnormal, 8..15 normal with the
// smallest exponent), so splitting a word takes a mask and a shift, no
// conversion.  A product of two digits is at most 225 in units of 2^-18, and a
// float accumulator of such sums is exact below 2^24 of them: 74565 terms.
// A chunk is a word's sixteen digit bytes: the low digits of bytes 0..7, then
// the high digits (digit e < 8 weighs 16^(2 e), digit 8 + b 16^(2 b + 1)).
#pragma once
#include "round_common.cuh"

#include <atomic>

namespace effsc {

__device__ __forceinline__ uint4 digits_of(u64 v) {
    const u32 w0 = (u32)v, w1 = (u32)(v >> 32), m = 0x0F0F0F0Fu;
    return make_uint4(w0 & m, w1 & m, (w0 >> 4) & m, (w1 >> 4) & m);
}
// 128-byte rows with the 128-byte swizzle: chunk c of row r.
__device__ __forceinline__ u32 swz128(u32 row, u32 chunk) { return row * 128 + ((chunk ^ (row & 7)) << 4); }

// Shared-memory matrix descriptor with the 128-byte swizzle: start address,
// bytes between 128-byte wide atoms, bytes between 8-row groups of an atom.
__device__ __forceinline__ u64 tc_desc(u32 addr, u32 atoms, u32 groups) {
    return (u64)((addr & 0x3FFFF) >> 4) | ((u64)(atoms >> 4) << 16) | ((u64)(groups >> 4) << 32) | (1ULL << 46) | (2ULL << 61);
}
// Instruction descriptor of kind::f8f6f4, e4m3 x e4m3 -> f32 (mn: both
// operands stored with the M / N index contiguous, else K).
__host__ __device__ constexpr u32 tc_idesc(u32 m, u32 n, bool mn) {
    return (1u << 4) | (mn ? (1u << 15) | (1u << 16) : 0u) | ((n >> 3) << 17) | ((m >> 4) << 24);
}
__device__ __forceinline__ void tc_mma_f8(u32 d, u64 a, u64 b, u32 idesc, u32 accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
// Arrive on `bar` when every MMA issued so far by this thread has finished.
__device__ __forceinline__ void tc_commit(u64* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Tensor memory, by one whole warp.
__device__ __forceinline__ void tc_alloc(u32* slot, u32 cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_dealloc(u32 addr, u32 cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// 16 columns of this warp's 32 tensor-memory lanes: issue, and wait for every
// load issued (the registers pass through the wait, so that nothing reads
// them before it).
__device__ __forceinline__ void tc_ld16(float (&f)[16], u32 addr) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=f"(f[0]), "=f"(f[1]), "=f"(f[2]), "=f"(f[3]), "=f"(f[4]), "=f"(f[5]), "=f"(f[6]), "=f"(f[7]),
                   "=f"(f[8]), "=f"(f[9]), "=f"(f[10]), "=f"(f[11]), "=f"(f[12]), "=f"(f[13]), "=f"(f[14]), "=f"(f[15])
                 : "r"(addr));
}
__device__ __forceinline__ void tc_wait_ld(float (&f)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+f"(f[0]), "+f"(f[1]), "+f"(f[2]), "+f"(f[3]), "+f"(f[4]), "+f"(f[5]), "+f"(f[6]), "+f"(f[7]),
                   "+f"(f[8]), "+f"(f[9]), "+f"(f[10]), "+f"(f[11]), "+f"(f[12]), "+f"(f[13]), "+f"(f[14]), "+f"(f[15])
                 :: "memory");
}
__device__ __forceinline__ void mbar_arrive(u64* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Tiles ahead of the register loads that a unit's 512 bytes are asked into L2.
constexpr int TC_PREFETCH = 2;
__device__ __forceinline__ void l2_prefetch(const void* p, u32 bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}
__device__ __forceinline__ void fence_async_shared() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }


// One word of digit products: 32 accumulator rows x 16 columns at `addr`, rows
// 16 q .. 16 q + 15 (lanes of half q) the digits of one word, the columns
// those of another; the two words' sum of products mod p in every lane of the
// half.
__device__ __forceinline__ u64 tc_row_sum(u32 addr, int lane) {
    const u32 d = lane & 15, sft = 4 * (d < 8 ? 2 * d : 2 * (d - 8) + 1);   // this row's weight 2^sft
    float f[16];
    tc_ld16(f, addr);
    tc_wait_ld(f);
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
    return v;
}

// ---------------------------------------------------------------------------
// Tiles of digit rows.  A tile is 128 items (groups of 2^NV table entries
// that one entry of the NV times folded table comes from) of two tables, an
// item a row of 16 x 2^NV digit bytes: one atom of [128 rows][128 bytes] per
// 8 values.  Rows 32 g + 16 h + p: item x = 16 g + .. of half h, the halves
// being the two items of a folded pair.  MSB: value v of item m is entry
// v N + m, halves m0 + x and m0 + x + H; LSB: value el of item o is entry
// o 2^NV + el, halves the items 2 x and 2 x + 1 of m0 .. m0 + 127.
// A unit is 16 bytes per lane of one warp; its two words are two items of one
// value (MSB) or two values of one item (LSB).  The row order within a half
// keeps the digit stores free of bank conflicts.
template <bool LSB, int NV>
struct TcTile {
    static constexpr int VALS = 1 << NV, ATOMS = VALS / 8;
    static constexpr u32 ATOM = 128 * 128, BYTES = 2 * ATOMS * ATOM;
    static constexpr int UNITS = 4 * VALS;
    static constexpr int LPI = VALS / 2, IPU = 32 / LPI;     // LSB: lanes per item, items per unit
    __device__ __forceinline__ static int table(int unit) { return unit / (2 * VALS); }
    __device__ __forceinline__ static u64 word(int unit, int lane, u64 m0, u64 H, u64 N) {
        const int u = unit % (2 * VALS);
        if (LSB) return (m0 + u * IPU + lane / LPI) * VALS + 2 * (lane % LPI);
        return (u64)(u >> 1) * N + m0 + (u & 1) * H + 2 * lane;
    }
    __device__ __forceinline__ static void store(char* stage, int unit, int lane, const ulonglong2& v) {
        const int u = unit % (2 * VALS);
        char* base = stage + table(unit) * ATOMS * ATOM;
        if (LSB) {
            const u32 o = u * IPU + lane / LPI, h = o & 1, k = o >> 1, q = lane % LPI;
            const u32 row = 32 * (k >> 4) + 16 * h + ((k & 15) ^ h);
            // NV = 4: a quarter warp stores one row's 16 chunks in two turns,
            // even ones of the first atom with odd ones of the second
            const u32 sel = NV == 4 ? q >> 2 : 0;
            base += (q >> 2) * ATOM;
            *(uint4*)(base + swz128(row, (2 * q + sel) & 7)) = digits_of(sel ? v.y : v.x);
            *(uint4*)(base + swz128(row, (2 * q + 1 - sel) & 7)) = digits_of(sel ? v.x : v.y);
        } else {
            const u32 val = u >> 1, row = 32 * (lane >> 3) + 16 * (u & 1) + (lane & 7);
            base += (val >> 3) * ATOM;
            *(uint4*)(base + swz128(row, val & 7)) = digits_of(v.x);
            *(uint4*)(base + swz128(row + 8, val & 7)) = digits_of(v.y);
        }
    }
    // Row 32 g + lane: which entry of the folded table (m0, H as above), and
    // the lane of the pair's other half.
    __device__ __forceinline__ static u64 entry(int g, int lane, u64 m0, u64 H) {
        const int h = lane >> 4, p = lane & 15;
        if (LSB) return m0 + 2 * (16 * g + (p ^ h)) + h;
        return m0 + 16 * g + 2 * (p & 7) + (p >> 3) + h * H;
    }
    static constexpr int PARTNER = LSB ? 17 : 16;
};

// This block's segment of a launch over many proofs, its arguments in `sa`.
__device__ __forceinline__ TcSeg tc_segment(const TcSeg* segs, u32 nsegs, const RoundArgs* args, RoundArgs& sa) {
    __shared__ u32 s_k;
    if (threadIdx.x == 0) {
        u32 lo = 0, hi = nsegs - 1;
        while (lo < hi) {
            const u32 mid = (lo + hi + 1) >> 1;
            if (segs[mid].first_block <= blockIdx.x) lo = mid; else hi = mid - 1;
        }
        s_k = lo;
    }
    __syncthreads();
    const u32 k = s_k;
    const u32* src = (const u32*)(args + k);
    u32* dst = (u32*)&sa;
    for (u32 w = threadIdx.x; w < sizeof(RoundArgs) / 4; w += blockDim.x) dst[w] = src[w];
    __syncthreads();
    return segs[k];
}

// The dynamic shared-memory limit is a per-device function attribute: set
// once per device (one bit each), safe when threads race to set it.
template <class K>
inline bool tc_allow_smem(K kernel, u32 bytes, std::atomic<uint64_t>& configured) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    const uint64_t bit = 1ull << (dev & 63);
    if (!(configured.load() & bit)) {
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess) return false;
        configured.fetch_or(bit);
    }
    return true;
}

}  // namespace effsc
