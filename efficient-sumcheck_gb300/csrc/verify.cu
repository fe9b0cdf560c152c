// verify.cu -- sumcheck_verify (src/verifier.rs:61-139) for many proofs at
// once: one warp per proof replays the proof's transcript (receive the wire
// values, absorb the hook bytes, squeeze the challenge); the claim follows
// from the EvalsInfty values:
//   h(1) = claim - h(0); h(inf) = recv[1] (degree >= 2) or h(1) - h(0);
//   q = [h(0), h(1) - h(inf), h(2) - 8 h(inf)] over {0, .., d-1};
//   claim = q(r) + h(inf) r^d,  q(r) by Lagrange interpolation.
// The final claims come back for the caller's oracle check (final_claim ==
// g(r)); for proofs made here that is the proof's final value.
#include "effsc_gpu.h"
#include "kernels.h"
#include "round_common.cuh"

#include <cstring>
#include <vector>

using namespace effsc;

int effsc_internal_ctx_device(const effsc_ctx* c);
cudaStream_t effsc_internal_ctx_stream(const effsc_ctx* c);
uint64_t effsc_internal_add_launches(uint64_t k);
void effsc_internal_tx_state(const effsc_transcript* t, void* out);
void* effsc_internal_pinned_get(effsc_ctx* c, size_t bytes);
void effsc_internal_pinned_put(effsc_ctx* c, void* p, size_t bytes);

namespace effsc {

struct VerifyArgs {
    const u64* claimed;       // field words per proof
    const u64* polys;         // field words per element, max(degree, 1) elements per row
    const u64* row_off;       // first row of proof i (n + 1 of them)
    const DevTranscript* tx;  // one per proof (state at the start)
    const uint8_t* hook;
    u32 hook_len;
    u32 degree;
    u32 field;
    u32 n;
    u64* challenges;          // field words per row (optional)
    u64* finals;              // field words per proof
};

// The round's update of the claim as an affine map, claim -> A claim + B.
__device__ __forceinline__ void verify_map(u32 d, const u64* w, const F3& r, F3& A, F3& B) {
    const F3 h0 = f3_make(w[0], w[1], w[2]);
    if (d == 0) {
        A = f3_zero();
        B = h0;
        return;
    }
    if (d == 1) {                      // claim = h0 + (claim - 2 h0) r
        A = r;
        B = f3_sub<true>(h0, f3_mul<true, true>(r, f3_add<true>(h0, h0)));
        return;
    }
    const F3 hinf = f3_make(w[3], w[4], w[5]), hs = f3_add<true>(h0, hinf);
    if (d == 2) {                      // h0 + r (claim - hs - h0) + hinf r^2
        A = r;
        B = f3_add<true>(h0, f3_mul<true, true>(r, f3_sub<true>(f3_mul<true, true>(r, hinf), f3_add<true>(hs, h0))));
        return;
    }
    // q2 = h(2) - 8 h(inf); Lagrange over {0, 1, 2}:
    // q(r) = q0 (r-1)(r-2)/2 - q1 r (r-2) + q2 r (r-1)/2, q1 = claim - hs
    F3 h8 = f3_add<true>(hinf, hinf);
    h8 = f3_add<true>(h8, h8);
    h8 = f3_add<true>(h8, h8);
    const F3 q2 = f3_sub<true>(f3_make(w[6], w[7], w[8]), h8);
    const F3 rm1 = f3_sub<true>(r, f3_make(1, 0, 0)), rm2 = f3_sub<true>(r, f3_make(2, 0, 0));
    const u64 inv2 = 0x7FFFFFFF80000001ULL;   // (p + 1) / 2
    const F3 t0 = f3_mul<true, true>(f3_mul<true, true>(rm1, rm2), h0);
    const F3 rr1 = f3_mul<true, true>(r, rm1), rr2 = f3_mul<true, true>(r, rm2);
    F3 half = f3_add<true>(t0, f3_mul<true, true>(rr1, q2));
    half = f3_make(gl_mul(half.c0, inv2), gl_mul(half.c1, inv2), gl_mul(half.c2, inv2));
    A = f3_sub<true>(f3_zero(), rr2);
    B = f3_add<true>(f3_add<true>(half, f3_mul<true, true>(rr2, hs)),
                     f3_mul<true, true>(hinf, f3_mul<true, true>(f3_mul<true, true>(r, r), r)));
}

// What bounds it is the longest proof's chain of permutations (2.2 us each):
// so nothing else is on it.  The wire words are read a round ahead, the
// transcript steps of 32 rounds run one after the other, and then each lane
// forms one round's affine map and five levels of composition give the claim
// (one lane updating the claim between the steps took 1 us a round).  256
// proofs of 10 to 22 rounds, the whole call from Python: 559 -> 446 us, with
// the blocks' allocations and copies taken out below.
constexpr int VERIFY_WARPS = 4;
__global__ void __launch_bounds__(32 * VERIFY_WARPS) k_verify_batch(VerifyArgs a) {
    __shared__ u64 s_wire[VERIFY_WARPS][32][9];
    __shared__ u64 s_chal[VERIFY_WARPS][32][3];
    __shared__ u64 s_gen[VERIFY_WARPS][12];
    __shared__ __align__(8) uint8_t s_scr[VERIFY_WARPS][64];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const u32 i = blockIdx.x * VERIFY_WARPS + wib;
    if (i >= a.n) return;
    const u32 d = a.degree, f = a.field;
    const int nw = (int)((d > 1 ? d : 1) * f);
    auto canon = [](u64 x) { return x >= GL_P ? x - GL_P : x; };
    const u64 row0 = a.row_off[i], rounds = a.row_off[i + 1] - row0;
    const u64* src = a.polys + row0 * nw;
    u64 next = lane < nw && rounds ? src[lane] : 0;
    WarpTx w = tx_load(a.tx + i, lane);
    const TxStream st = tx_stream(nw, a.hook, a.hook_len, lane);
    F3 claim = f3_zero();
    claim.c0 = canon(a.claimed[(u64)i * f]);
    if (f == 3) {
        claim.c1 = canon(a.claimed[(u64)i * 3 + 1]);
        claim.c2 = canon(a.claimed[(u64)i * 3 + 2]);
    }
    const int at = f == 3 ? lane : 3 * lane;      // the wire word's place among elements of three
    for (int k = lane; k < 32 * 9; k += 32) s_wire[wib][0][k] = 0;
    __syncwarp();
    for (u64 c0 = 0; c0 < rounds; c0 += 32) {
        const u32 cnt = rounds - c0 < 32 ? (u32)(rounds - c0) : 32;
        for (u32 j = 0; j < cnt; j++) {
            const u64 wire = canon(next);
            if (lane < nw && c0 + j + 1 < rounds) next = src[(c0 + j + 1) * nw + lane];
            if (lane < nw) s_wire[wib][j][at] = wire;
            const u64 r = tx_step(w, st, nw, (int)f, wire, a.hook, a.hook_len, lane, s_gen[wib], s_gen[wib] + 9, s_scr[wib]);
            if (lane < 3) s_chal[wib][j][lane] = r;
        }
        __syncwarp();
        if (a.challenges)
            for (u32 k = lane; k < cnt * f; k += 32) a.challenges[(row0 + c0) * f + k] = s_chal[wib][k / f][k % f];
        F3 A = f3_make(1, 0, 0), B = f3_zero();
        if ((u32)lane < cnt) verify_map(d, s_wire[wib][lane], f3_make(s_chal[wib][lane][0], s_chal[wib][lane][1], s_chal[wib][lane][2]), A, B);
        __syncwarp();
#pragma unroll 1
        for (int o = 1; o < 32; o <<= 1) {        // lanes l .. l + o - 1, then l + o .. l + 2 o - 1
            auto up = [&](const F3& v) {
                return f3_make(__shfl_down_sync(0xffffffffu, v.c0, o), __shfl_down_sync(0xffffffffu, v.c1, o),
                               __shfl_down_sync(0xffffffffu, v.c2, o));
            };
            const F3 A2 = up(A), B2 = up(B);
            B = f3_add<true>(f3_mul<true, true>(A2, B), B2);
            A = f3_mul<true, true>(A2, A);
        }
        claim = f3_add<true>(f3_mul<true, true>(A, claim), B);      // lane 0's
    }
    if (lane == 0) {
        a.finals[(u64)i * f] = claim.c0;
        if (f == 3) {
            a.finals[(u64)i * 3 + 1] = claim.c1;
            a.finals[(u64)i * 3 + 2] = claim.c2;
        }
    }
}

}  // namespace effsc

// Blocks of powers of two from 64 KB, so that calls of similar size share
// them; above 4 MB pinning costs more than the copies it saves.
constexpr size_t VERIFY_BLOCK_MIN = 64 << 10, VERIFY_IN_PLACE = 4 << 20;

#define VCK(call)                                                                                           \
    do {                                                                                                    \
        cudaError_t e_ = (call);                                                                            \
        if (e_ != cudaSuccess) { rc = effsc_set_error(EFFSC_CUDA_ERROR, "%s: %s", #call, cudaGetErrorString(e_)); goto done; } \
    } while (0)

extern "C" int effsc_verify_batch(effsc_ctx* ctx, int field, size_t n, const uint64_t* claimed_sums, int degree,
                                  const uint32_t* num_rounds, const effsc_transcript* const* transcripts,
                                  const uint8_t* hook, size_t hook_len, const uint64_t* round_polys,
                                  uint64_t* challenges, uint64_t* final_claims) {
    if (!ctx || !claimed_sums || !num_rounds || !transcripts || !final_claims || (hook_len && !hook))
        return effsc_set_error(EFFSC_INVALID_ARG, "NULL argument");
    if (field != EFFSC_FP && field != EFFSC_FP3) return effsc_set_error(EFFSC_INVALID_ARG, "bad field");
    if (degree < 0 || degree > 3) return effsc_set_error(EFFSC_UNSUPPORTED, "device verification handles degree 0..3");
    if (hook_len >= (1ull << 32) || n >= (1ull << 32)) return effsc_set_error(EFFSC_INVALID_ARG, "hook or batch too large");
    if (!n) return EFFSC_OK;
    const int dev = effsc_internal_ctx_device(ctx);
    cudaStream_t s = effsc_internal_ctx_stream(ctx);
    if (cudaSetDevice(dev) != cudaSuccess) return effsc_set_error(EFFSC_CUDA_ERROR, "cudaSetDevice");
    const u32 nw = degree > 1 ? degree : 1;
    size_t rows = 0;
    for (size_t i = 0; i < n; i++) {
        rows += num_rounds[i];
        if (!transcripts[i]) return effsc_set_error(EFFSC_INVALID_ARG, "transcript %zu is NULL", i);
    }
    if (rows && !round_polys) return effsc_set_error(EFFSC_INVALID_ARG, "round_polys is NULL");
    // One block of host memory, words: row offsets, claims, polynomials, hook,
    // transcripts, then the challenges and final claims.  Up to
    // VERIFY_IN_PLACE the kernel reads and writes it there (pinned), a round
    // ahead of its use; a larger one is copied to the device and back.
    constexpr size_t TXW = (sizeof(DevTranscript) + 7) / 8;
    const size_t o_claims = n + 1, o_polys = o_claims + n * field, o_hook = o_polys + rows * nw * field;
    const size_t o_tx = o_hook + (hook_len + 7) / 8, o_out = o_tx + n * TXW, o_fin = o_out + (challenges ? rows * field : 0);
    const size_t words = o_fin + n * field;
    size_t bytes = VERIFY_BLOCK_MIN;
    while (bytes < words * 8) bytes *= 2;
    bool in_place = bytes <= VERIFY_IN_PLACE;
    std::vector<u64> big;
    u64* h = nullptr;
    u64* dv = nullptr;
    if (in_place) {
        h = (u64*)effsc_internal_pinned_get(ctx, bytes);
        in_place = h != nullptr;
    }
    if (!in_place) {
        big.resize(words);
        h = big.data();
    }
    int rc = EFFSC_OK;
    h[0] = 0;
    for (size_t i = 0; i < n; i++) {
        DevTranscript* t = (DevTranscript*)(h + o_tx + i * TXW);
        h[i + 1] = h[i] + num_rounds[i];
        effsc_internal_tx_state(transcripts[i], t);
        if ((int)t->deg != field) { rc = effsc_set_error(EFFSC_INVALID_ARG, "transcript %zu: wrong field or kind", i); goto done; }
    }
    memcpy(h + o_claims, claimed_sums, n * field * 8);
    if (rows) memcpy(h + o_polys, round_polys, rows * nw * field * 8);
    if (hook_len) memcpy(h + o_hook, hook, hook_len);
    {
        u64* base = h;
        if (in_place) {
            VCK(cudaHostGetDevicePointer((void**)&base, h, 0));
        } else {
            VCK(cudaMallocAsync((void**)&dv, words * 8, s));
            VCK(cudaMemcpyAsync(dv, h, o_out * 8, cudaMemcpyHostToDevice, s));
            base = dv;
        }
        VerifyArgs va;
        va.claimed = base + o_claims; va.polys = base + o_polys; va.row_off = base; va.tx = (const DevTranscript*)(base + o_tx);
        va.hook = (const uint8_t*)(base + o_hook); va.hook_len = (u32)hook_len; va.degree = (u32)degree; va.n = (u32)n;
        va.field = (u32)field; va.challenges = challenges ? base + o_out : nullptr; va.finals = base + o_fin;
        k_verify_batch<<<(unsigned)((n + VERIFY_WARPS - 1) / VERIFY_WARPS), 32 * VERIFY_WARPS, 0, s>>>(va);
        effsc_internal_add_launches(1);
        VCK(cudaGetLastError());
    }
    if (!in_place) VCK(cudaMemcpyAsync(h + o_out, dv + o_out, (words - o_out) * 8, cudaMemcpyDeviceToHost, s));
    VCK(cudaStreamSynchronize(s));
    memcpy(final_claims, h + o_fin, n * field * 8);
    if (challenges && rows) memcpy(challenges, h + o_out, rows * field * 8);
done:
    if (dv) cudaFreeAsync(dv, s);
    if (in_place) effsc_internal_pinned_put(ctx, h, bytes);
    return rc;
}
