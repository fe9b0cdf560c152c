// k_ml_phase.cu -- a Multilinear proof from two reads of its base table.
//
// A round sends the sum of the lower half alone (src/provers/multilinear.rs:
// 52-61), and sums are linear: with the variables bound first, b, and the
// rest, c, the first rounds are Multilinear rounds on T(b) = sum_c p(b, c), a
// table of half the variables.  The rest run on p folded with all those
// challenges at once, sum_b e(b) p(b, c) with the eq weights e (k_eqf_tc.cu,
// k_eqf.cu).  Both are a tail's size, so the proof is two reads of p and two
// tails, where rounds of folding wrote half of the table and read it again,
// or held it in one cluster from the start.
//
// MSB: b is the high half of the index, T a sum along rows; LSB: the low half,
// a sum down columns.  Memory bounds both reads from 2^24 entries on; below, the
// two tails are three quarters of the time (20 rounds of 3.4 us).  A call, Fp,
// 2^20 entries: 127 -> 111 us (LSB 143 -> 114; 101 with the present
// permutation); Fp3, 2^25: 448 -> 250 (LSB 618 -> 255).
#include "round_common.cuh"

namespace effsc {

// T[b] = sum of row b (m entries), a block per row.
__global__ void __launch_bounds__(TPB) k_ml_rows(const u64* p, u64 m, u64* T) {
    chain_enter();
    __shared__ uint4 s_p[NWARP];
    const u64* row = p + blockIdx.x * m;
    Acc s = acc_zero();
#pragma unroll 8
    for (u64 c = threadIdx.x; c < m; c += TPB) acc_add64(s, __ldcs(row + c));
    const uint4 q = warp_sum_pieces(acc_reduce(s));
    if ((threadIdx.x & 31) == 0) s_p[threadIdx.x >> 5] = q;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint4 t = s_p[0];
        for (int w = 1; w < NWARP; w++) { t.x += s_p[w].x; t.y += s_p[w].y; t.z += s_p[w].z; }
        T[blockIdx.x] = join_pieces(t);
    }
}

// part[3 (split m + b)] = sum over the split's rows c of p[c m + b].
__global__ void __launch_bounds__(TPB) k_ml_cols(const u64* p, u64 m, u64 per, u64 tiles, u64* part) {
    chain_enter();
    const u64 tile = blockIdx.x % tiles, split = blockIdx.x / tiles, b = tile * TPB + threadIdx.x;
    if (b >= m) return;
    const u64* q = p + split * per * m + b;
    Acc s = acc_zero();
#pragma unroll 8
    for (u64 c = 0; c < per; c++) acc_add64(s, __ldcs(q + c * m));
    part[3 * (split * m + b)] = acc_reduce(s);
}

bool launch_ml_rows(const u64* p, u64 m, u64 rows, u64* T, cudaStream_t s) {
    return launch_chain(k_ml_rows, (int)rows, TPB, 0, s, p, m, T);
}
bool launch_ml_cols(const u64* p, u64 m, u64 rows, u64 splits, u64* part, u64* T, cudaStream_t s) {
    const u64 tiles = (m + TPB - 1) / TPB;
    if (!launch_chain(k_ml_cols, (int)(tiles * splits), TPB, 0, s, p, m, rows / splits, tiles, part)) return false;
    launch_eqf_sum(part, m, splits, 1, T, nullptr, nullptr, s);
    return true;
}

}  // namespace effsc
