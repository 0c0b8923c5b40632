// verify_body.cuh -- one MAYO verify (reference src/verify.cu:9-212) on one CTA, or on a cluster of
// CTAs where a batch is too small to fill the GPU; shared by the batched verify kernels and the
// persistent work-queue kernel.
//
// U_ij = s_i^T P s_j (+ symmetric term) over the expanded public key P = [[P1, P2], [0, P3]] in two
// steps of the same product (quad.cuh): T_j[r] = sum_c P[r][c] s_j[c] for the key's quads of rows,
// then X_ij = sum_r s_i[r] T_j[r] over the quads, both with warps that take chunks of 32 units
// from a counter.  Warp 0 first hashes digest = SHAKE256(M) and t = SHAKE256(digest || salt).
// y = sum z^l U_l is then collected by all warps and compared with t.
#pragma once

#include "launch_util.cuh"
#include "quad.cuh"

namespace mayo {

template <int SET, int CL = 1>
struct VerifyCfg {
    using S = Set<SET>;
    using A = QuadAcc<S::k>;
    static constexpr int J = S::k, NQ = QuadCfg<SET>::NQ, ST = A::ST;
    static constexpr int QN = (S::n + 3) / 4;  // quads of rows
    // The quads are dealt out to the CTAs of a cluster, quad Q to CTA Q % NP, so that each has long
    // and short rows.
    static constexpr int NP = CL;
    static constexpr int QL = (QN + NP - 1) / NP;
    static constexpr int UL = QL * NQ;               // units of a part
    static constexpr int CH = (UL + 31) / 32;        // chunks of 32 units
    static constexpr int CW = CL > 1 ? 8 : (SET == 1 ? 4 : SET == 2 ? 3 : 8);  // warps
    static constexpr int NT = 32 * CW;
    // column ranges per chunk (more items than warps where a cluster leaves few chunks per CTA)
    static constexpr int PC = CL > 1 ? (2 * CW + CH - 1) / CH : 1;
    static constexpr int CH2 = (J * NQ + 31) / 32;   // chunks of (j, word) pairs
    static constexpr int P2 = CL == 1 && SET == 5 ? 1 : (CW + CH2 - 1) / CH2;  // quad ranges of each
    // Warps, CTAs per SM and columns loaded ahead.  Registers for two columns ahead beat more warps
    // where nine accumulators per vector leave few: MAYO_3 one CTA of 8 warps (241 registers) 0.381 us
    // per instance at 2,072, of 7 0.406, of 12 (168, one ahead) 0.539, two of 4 with T in two halves
    // 0.428; MAYO_5 8 warps 0.752, one ahead 0.844, 11 (168) 0.846.  MAYO_1: three CTAs of 4, one
    // ahead 0.153 (two 0.180; two CTAs, two ahead 0.169); MAYO_2 0.064 (one 0.067).
    static constexpr int D = SET == 1 ? 1 : 2;
    static constexpr int MINB = CL > 1 ? 1 : (SET == 1 ? 3 : SET == 2 ? 6 : 1);
    static constexpr size_t off_masks = 0;
    static constexpr size_t sz_masks = (size_t)S::n * ST * 16;
    static constexpr size_t sz_mask2 = (size_t)QL * ST * 16, sz_upk = pad16((size_t)S::pairs * NQ * 4);
    // the second step's masks and U take the first one's masks' place
    static constexpr size_t off_mask2 = 0, off_upk = sz_mask2;
    static_assert(sz_mask2 + sz_upk <= sz_masks, "second-step masks and U fit");
    static constexpr size_t off_T = sz_masks;
    static constexpr size_t off_yext = off_T + (size_t)J * CH * 32 * 16;
    static constexpr size_t off_sig = off_yext + 128;
    static constexpr size_t off_key = off_sig + pad16(S::sig);
    static constexpr size_t off_t = off_key + pad16(S::digest + S::sk);
    static constexpr size_t off_ctr = off_t + pad16(NQ * 4);
    static constexpr size_t total = off_ctr + 16;
};

// Verify one instance; every thread of the CTA (VerifyCfg::NT of them), or of every CTA of the
// cluster (rank = this CTA's), must call it.  Writes 0 (accept) or 1 (reject) to *res.  `smem` holds
// VerifyCfg<SET, CL>::total bytes, at the same address in every CTA of a cluster.  HASHED: the message's
// digest is at off_key already (the caller's stores need no barrier), `msg` and `mlen` are not used.
template <int SET, int CL = 1, bool HASHED = false>
__device__ __forceinline__ void verify_instance(uint8_t *smem, int tid, const uint8_t *epk, const uint8_t *msg,
                                                uint32_t mlen, const uint8_t *sig, uint8_t *res, int rank = 0) {
    using S = Set<SET>;
    using C = VerifyCfg<SET, CL>;
    constexpr int J = C::J, NQ = C::NQ, NT = C::NT, CW = C::CW, ULP = C::CH * 32;
    uint4 *masks = reinterpret_cast<uint4 *>(smem + C::off_masks);
    uint4 *mask2 = reinterpret_cast<uint4 *>(smem + C::off_mask2);
    uint32_t *upk = reinterpret_cast<uint32_t *>(smem + C::off_upk);  // [l][NQ]
    uint4 *T = reinterpret_cast<uint4 *>(smem + C::off_T);            // [j][unit]
    uint32_t *yext = reinterpret_cast<uint32_t *>(smem + C::off_yext);
    uint8_t *s_sig = smem + C::off_sig;
    uint8_t *s_key = smem + C::off_key;
    uint8_t *s_t = smem + C::off_t;
    int *s_next = reinterpret_cast<int *>(smem + C::off_ctr);
    const int warp = tid >> 5, lane = tid & 31;

    for (int i = tid; i < S::sig; i += NT) s_sig[i] = sig[i];
    for (int i = tid; i < NQ * 4; i += NT) s_t[i] = 0;
    if (tid < 32) yext[tid] = 0;
    if (tid == 0) *s_next = 0;
    __syncthreads();

    // scalar c of s_j (src/verify.cu:62-70)
    auto scalar = [&](int c, int j) {
        const int q = j * S::n + c;
        return (uint32_t)(s_sig[q >> 1] >> ((q & 1) * 4)) & 0xFu;
    };
    build_masks9<J>(reinterpret_cast<uint32_t *>(masks), S::n, tid, NT, scalar);
    const uint32_t mis = (uint32_t)(reinterpret_cast<uintptr_t>(epk) & 3);
    const uint32_t *base4 = reinterpret_cast<const uint32_t *>(epk - mis);
    if constexpr (CL == 1) {  // every row's first columns of P1, then P2 and P3, while the masks are built
        for (int r = tid; r < S::v; r += NT) PubRows<SET>::row_ahead(base4, mis, r, r);
        l2_prefetch_range(base4, mis + S::p1, S::epk - S::p1, tid, NT);
    }

    const int part = rank;
    auto quad_scalar = [&](int t, int i, int j) {
        const int c = 4 * (part + t * C::NP) + i;
        return c < S::n ? scalar(c, j) : 0u;
    };
    if constexpr (C::PC > 1) {
        for (int i = tid; i < J * ULP; i += NT) T[i] = make_uint4(0, 0, 0, 0);
    }
    __syncthreads();
    if (rank == 0 && warp == 0) {  // digest and target t (src/verify.cu:37-48)
        WarpKeccak wk;
        wk.setup(lane);
        if constexpr (!HASHED) warp_shake<136>(s_key, S::digest, msg, mlen, wk, lane);
        for (int i = lane; i < S::sk; i += 32) s_key[S::digest + i] = s_sig[S::k * S::n / 2 + i];
        __syncwarp();
        warp_shake<136>(s_t, S::menc, s_key, S::digest + S::sk, wk, lane);
    }
    // ---- T_j[r] = sum_c P[r][c] s_j[c]: chunks of 32 units, the longest first ----
    for (;;) {
        const int item = warp_next(s_next, lane);
        if (item >= C::CH * C::PC) break;
        const int chunk = item / C::PC, piece = item - chunk * C::PC;
        const int u = chunk * 32 + lane, t = u / NQ, q = u - t * NQ;
        const int r0 = 4 * (part + t * C::NP);
        const int qmin = part + (chunk * 32 / NQ) * C::NP, qmax = part + ((chunk * 32 + 31) / NQ) * C::NP;
        const int c_lo = min(4 * qmin, S::n), c_chk = 4 * min(qmax, C::QN - 1) + 4;
        const int len = S::n - c_lo;
        QuadAcc<J> acc;
        acc.zero();
        const int tl = chunk * 32 / NQ + (lane >> 2);
        const PubRows<SET> rows{mis, (uint32_t)(4 * q), r0,
                                tl <= (chunk * 32 + 31) / NQ ? 4 * (part + tl * C::NP) + (lane & 3) : S::n};
        const int ca = c_lo + len * piece / C::PC, cb = c_lo + len * (piece + 1) / C::PC;
#pragma unroll 1
        for (int seg = 0; seg < 2; seg++)  // P1's columns, then P2's and P3's
            quad_columns<SET, J, true, C::D>(acc, rows, base4, QuadCfg<SET>::bytes(q), seg ? max(ca, S::v) : ca,
                                       seg ? cb : min(cb, S::v), c_chk, masks, mis == 0);
        const uint32_t rm = quad_row_mask(r0, S::n);
#pragma unroll
        for (int j = 0; j < J; j++) {
            const G4 v = g4_and(acc.fold(j), rm);
            if constexpr (C::PC > 1) g4_atomic_xor(T + j * ULP + u, v);
            else g4_st(T + j * ULP + u, v);
        }
    }
    __syncthreads();
    build_quad_masks9<J>(reinterpret_cast<uint32_t *>(mask2), C::QL, tid, NT, quad_scalar);
    for (int i = tid; i < S::pairs * NQ; i += NT) upk[i] = 0;
    __syncthreads();
    // ---- X_ij = sum_r s_i[r] T_j[r], packed into U_l ----
    quad_pairs<SET, C>(T, ULP, mask2, upk, 0, warp, lane, [](int a, int b) { return pair_ell(a, b, J); });
    __syncthreads();
    if constexpr (CL > 1) {  // the ranks' parts of U meet in rank 0
        cluster_barrier();
        if (rank == 0) {
            for (int i = tid; i < S::pairs * NQ; i += NT) upk[i] = xor_cluster<CL>(upk + i);
        }
        cluster_barrier();  // no CTA leaves while rank 0 reads its shared memory
        if (rank != 0) return;
    }
    y_accumulate<SET>(upk, yext, warp, CW, lane);
    __syncthreads();
    if (warp == 0) {  // compare y with t (src/verify.cu:185-211)
        const uint32_t y = y_fold<SET>(yext, lane);
        const uint32_t tw = lane < NQ ? reinterpret_cast<const uint32_t *>(s_t)[lane] : 0u;
        const bool eq = __all_sync(0xffffffffu, y == tw);
        if (lane == 0) *res = eq ? 0 : 1;
    }
}

}  // namespace mayo
