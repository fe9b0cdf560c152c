// k_gkr_phase.cu -- a whole GkrProver proof from two reads of the gate tables.
//
// f(b, c) = add(b, c) (W(b) + W(c)) + mult(b, c) W(b) W(c) is linear in add and
// mult, and each of them meets only one witness variable at a time, so the
// 2k rounds (src/provers/gkr.rs:105-190) are InnerProduct rounds on tables of
// 2n entries, n = 2^k = |w|, where the gate tables hold n^2:
//   rounds 0 .. k-1 bind b.  With
//     A(b) = sum_c add(b, c),  B(b) = sum_c add(b, c) W(c),  M(b) = sum_c mult(b, c) W(c)
//   the sum is sum_b W(b) (A(b) + M(b)) + 1 B(b): the inner product of
//   F = (W(b), 1) and G = (A(b) + M(b), B(b)), the pair's place the last
//   variable, which is never bound;
//   rounds k .. 2k-1 bind c.  With the weights e(b) = eq(r, b) of the first k
//   challenges, a(c) = sum_b e(b) add(b, c), m(c) = sum_b e(b) mult(b, c) and
//   w = W(r), the sum is the inner product of F = (w W(c), w + W(c)) and
//   G = (m(c), a(c)), whose last fold leaves mult and add themselves.
// The wire [q(0), q(inf)] is the same two field elements: x^2's coefficient
// is sum dF dG.  All sums are exact, so nothing depends on their order.
//
// Folding the gate tables round by round moved 7.5 n^2 words (k = 12: 692 us
// of kernels); this reads them twice, 71 us each on the tensor cores
// (k_eqf_tc.cu), plus two tails of 63 us: 294 us.  The tails are one warp's
// latency, the reads two thirds of the copy rate.  Up to n = 1024 the sums run
// here on the integer pipes, a warp per row and eight columns a block: their
// tables fit L2 and a tensor-core block's start and end cost more than they do
// (k = 9, a whole proof: 145 us against 172; k = 10: 177 against 191; beyond,
// 1 : 1 at best and an eq weight per row in every block).
#include "round_common.cuh"

namespace effsc {

__device__ __forceinline__ u64 gkr_sum_at(const GkrSums& s, u64 m, int c) {
    const u64* p = s.p + 3 * m + c;
    u64 v = p[0];
    for (u32 i = 1; i < s.splits; i++) v = gl_add(v, p[i * 3 * s.n]);
    return v;
}

// F = (W, 1), G = (A + M, B) from the weighted row sums: of add with the
// weights (W, 1) and of mult with W.
__global__ void __launch_bounds__(TPB) k_gkr_terms_b(GkrSums add, GkrSums mult, const u64* W, u64* F, u64* G) {
    chain_enter();
    const u64 b = (u64)blockIdx.x * TPB + threadIdx.x;
    if (b >= add.n) return;
    ((ulonglong2*)F)[b] = make_ulonglong2(W[b], 1);
    ((ulonglong2*)G)[b] = make_ulonglong2(gl_add(gkr_sum_at(add, b, 1), gkr_sum_at(mult, b, 0)), gkr_sum_at(add, b, 0));
}

// The same from the gate tables, a warp per row.
__global__ void __launch_bounds__(TPB) k_gkr_rows(const u64* add, const u64* mult, const u64* W, u32 n, u64* F, u64* G) {
    chain_enter();
    const u32 b = blockIdx.x * NWARP + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (b >= n) return;
    Acc h = acc_zero(), s = acc_zero();
#pragma unroll 4
    for (u32 c = lane; c < n; c += 32) {
        const u64 x = add[(u64)b * n + c], w = W[c];
        acc_add64(h, x);
        acc_mac(h, mult[(u64)b * n + c], w);
        acc_mac(s, x, w);
    }
    const uint4 ph = warp_sum_pieces(acc_reduce(h)), ps = warp_sum_pieces(acc_reduce(s));
    if (lane == 0) {
        ((ulonglong2*)F)[b] = make_ulonglong2(W[b], 1);
        ((ulonglong2*)G)[b] = make_ulonglong2(join_pieces(ph), join_pieces(ps));
    }
}

// F = (w W, w + W) and G = (m, a), component q of a table in the plane q (2n
// words each); wb: W(r), component q at wb[2 q].
template <int FW>
__device__ __forceinline__ void gkr_put_c(const u64* wb, u64 Wc, u64 n, u64 c, const F3& m, const F3& a, u64* F, u64* G) {
#pragma unroll
    for (int q = 0; q < FW; q++) {
        const u64 w = wb[2 * q];
        ((ulonglong2*)(F + 2 * n * q))[c] = make_ulonglong2(gl_mul(w, Wc), q ? w : gl_add(w, Wc));
        ((ulonglong2*)(G + 2 * n * q))[c] =
            make_ulonglong2(q == 0 ? m.c0 : q == 1 ? m.c1 : m.c2, q == 0 ? a.c0 : q == 1 ? a.c1 : a.c2);
    }
}
template <int FW>
__global__ void __launch_bounds__(TPB) k_gkr_terms_c(GkrSums add, GkrSums mult, const u64* W, const u64* wb, u64* F, u64* G) {
    chain_enter();
    const u64 c = (u64)blockIdx.x * TPB + threadIdx.x;
    if (c >= add.n) return;
    F3 m = f3_zero(), a = f3_zero();
    m.c0 = gkr_sum_at(mult, c, 0);
    a.c0 = gkr_sum_at(add, c, 0);
    if (FW == 3) {
        m.c1 = gkr_sum_at(mult, c, 1); m.c2 = gkr_sum_at(mult, c, 2);
        a.c1 = gkr_sum_at(add, c, 1); a.c2 = gkr_sum_at(add, c, 2);
    }
    gkr_put_c<FW>(wb, W[c], add.n, c, m, a, F, G);
}

// The same from the gate tables: eight columns a block, thread = (column, one
// of 32 groups of rows); each block forms the n <= GKR_SMALL weights itself.
template <int FW>
__global__ void __launch_bounds__(TPB) k_gkr_cols(const u64* add, const u64* mult, const u64* W, const u64* wb,
                                                  const u64* chals, u32 k, u64* F, u64* G) {
    chain_enter();
    __shared__ u64 s_e[FW][GKR_SMALL];
    __shared__ uint4 s_p[NWARP][8][2 * FW];
    const u32 n = 1u << k, t = threadIdx.x, lane = t & 31, warp = t >> 5;
    for (u32 b = t; b < n; b += TPB) {
        F3 e = f3_make(1, 0, 0);
        for (u32 j = 0; j < k; j++) {
            const F3 r = f3_make(chals[3 * j], chals[3 * j + 1], chals[3 * j + 2]);
            e = f3_mul<FW == 3, FW == 3>(e, ((b >> (k - 1 - j)) & 1) ? r : f3_sub<FW == 3>(f3_make(1, 0, 0), r));
        }
        s_e[0][b] = e.c0;
        if constexpr (FW == 3) { s_e[1][b] = e.c1; s_e[2][b] = e.c2; }
    }
    __syncthreads();
    const u32 c = blockIdx.x * 8 + (t & 7);
    Acc s[2 * FW];
#pragma unroll
    for (int i = 0; i < 2 * FW; i++) s[i] = acc_zero();
    if (c < n)
#pragma unroll 4
        for (u32 b = t >> 3; b < n; b += TPB / 8) {
            const u64 x = mult[(u64)b * n + c], y = add[(u64)b * n + c];
#pragma unroll
            for (int q = 0; q < FW; q++) {
                acc_mac(s[q], s_e[q][b], x);
                acc_mac(s[FW + q], s_e[q][b], y);
            }
        }
#pragma unroll
    for (int i = 0; i < 2 * FW; i++) {
        u64 v = acc_reduce(s[i]);
        v = gl_add(v, __shfl_xor_sync(0xffffffffu, v, 8));
        v = gl_add(v, __shfl_xor_sync(0xffffffffu, v, 16));
        if (lane < 8) s_p[warp][lane][i] = make_uint4((u32)v & 0x3FFFFFu, (u32)(v >> 22) & 0x3FFFFFu, (u32)(v >> 44), 0);
    }
    __syncthreads();
    if (t < 8 && c < n) {
        u64 v[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
        for (int i = 0; i < 2 * FW; i++) {
            uint4 p = s_p[0][t][i];
            for (int w = 1; w < NWARP; w++) {
                const uint4 q = s_p[w][t][i];
                p.x += q.x; p.y += q.y; p.z += q.z;
            }
            v[FW == 3 ? i : 3 * i] = join_pieces(p);
        }
        gkr_put_c<FW>(wb, W[c], n, c, f3_make(v[0], v[1], v[2]), f3_make(v[3], v[4], v[5]), F, G);
    }
}

// add, mult, W_b, W_c at the point, from the two tails' last tables (two
// entries a component): out[t][q] and the read-back entries.
__global__ void k_gkr_finish(const u64* fb, const u64* fc, const u64* gc, int fw, GkrFinish o) {
    chain_enter();
    const int q = threadIdx.x;
    if (q >= 3) return;
    u64 v[4] = {0, 0, 0, 0};
    if (q < fw) {
        v[0] = gc[2 * q + 1];
        v[1] = gc[2 * q];
        v[2] = fb[2 * q];
        v[3] = gl_sub(fc[2 * q + 1], v[2]);
    }
    for (int t = 0; t < 4; t++) {
        if (q < fw) o.out[t][q][0] = v[t];
        o.first[3 * t + q] = v[t];
    }
}

bool launch_gkr_terms_b(const GkrSums& add, const GkrSums& mult, const u64* W, u64* F, u64* G, cudaStream_t s) {
    return launch_dep(k_gkr_terms_b, (int)((add.n + TPB - 1) / TPB), TPB, 0, s, add, mult, W, F, G);
}
bool launch_gkr_rows(const u64* add, const u64* mult, const u64* W, u32 n, u64* F, u64* G, cudaStream_t s) {
    return launch_dep(k_gkr_rows, (int)((n + NWARP - 1) / NWARP), TPB, 0, s, add, mult, W, n, F, G);
}
bool launch_gkr_terms_c(int fw, const GkrSums& add, const GkrSums& mult, const u64* W, const u64* wb, u64* F, u64* G,
                        cudaStream_t s) {
    const int g = (int)((add.n + TPB - 1) / TPB);
    return fw == 3 ? launch_dep(k_gkr_terms_c<3>, g, TPB, 0, s, add, mult, W, wb, F, G)
                   : launch_dep(k_gkr_terms_c<1>, g, TPB, 0, s, add, mult, W, wb, F, G);
}
bool launch_gkr_cols(int fw, const u64* add, const u64* mult, const u64* W, const u64* wb, const u64* chals, u32 k, u64* F,
                     u64* G, cudaStream_t s) {
    const int g = ((1 << k) + 7) / 8;
    return fw == 3 ? launch_dep(k_gkr_cols<3>, g, TPB, 0, s, add, mult, W, wb, chals, k, F, G)
                   : launch_dep(k_gkr_cols<1>, g, TPB, 0, s, add, mult, W, wb, chals, k, F, G);
}
bool launch_gkr_finish(int fw, const u64* fb, const u64* fc, const u64* gc, const GkrFinish& o, cudaStream_t s) {
    return launch_dep(k_gkr_finish, 1, 32, 0, s, fb, fc, gc, fw, o);
}

}  // namespace effsc
