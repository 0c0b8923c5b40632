// keygen_body.cuh -- P3 of a keypair (reference src/keypair.cu:55-120) and L of an expanded
// secret key (src/expandsk.cu:37-80) on one CTA or a cluster of CTAs, shared by the batched kernels
// and the persistent work-queue kernel.  Both are products of the key's quads with O (quad.cuh).
#pragma once

#include "launch_util.cuh"
#include "quad.cuh"

namespace mayo {

// P3 = Upper(O^T T), T = P1 O + P2: the rows of P1 as in VerifyCfg, then T's quads with O again.
template <int SET, int CL_ = 1, int CW_ = 0>
struct KeyCfg {
    using S = Set<SET>;
    static constexpr int CL = CL_, J = S::o, NQ = QuadCfg<SET>::NQ, ST = QuadAcc<J>::ST;
    static constexpr int QN = (S::v + 3) / 4;
    static constexpr int NP = CL;
    static constexpr int QL = (QN + NP - 1) / NP;
    static constexpr int CH = (QL * NQ + 31) / 32;
    // Warps and CTAs per SM, keypairs at 2,072 (us per instance): MAYO_1 three CTAs of four warps 0.321
    // against 0.330 with four CTAs (128 registers, spills); MAYO_2 (153 accumulators) two warps 0.312
    // against 0.322 with four and 0.486 with three CTAs of three warps (spills); MAYO_3 two CTAs of
    // six warps (168 registers, a few words spilled) 0.796 against 0.809 with four warps and two columns
    // ahead; beside a faster expansion 0.698 against 0.729 with eight warps in one CTA; MAYO_5 one CTA of
    // eight warps, two columns ahead, 1.55 against 1.69 with eleven, one ahead.
    static constexpr int CW = CW_ ? CW_ : CL > 1 ? 8 : (SET == 1 ? 4 : SET == 2 ? 2 : SET == 3 ? 6 : 8);
    static constexpr int NT = 32 * CW;
    static constexpr int PC = CL > 1 ? (2 * CW + CH - 1) / CH : 1;
    static constexpr int CH2 = (J * NQ + 31) / 32;
    static constexpr int P2 = CH2 >= CW || (CL == 1 && SET == 5) ? 1 : (CW + CH2 - 1) / CH2;
    static constexpr int D = SET == 5 ? 2 : 1;  // columns loaded ahead
    static constexpr int MINB = CL > 1 ? 1 : (SET == 1 ? 3 : SET == 5 ? 1 : 2);
    static constexpr int TRI = S::o * (S::o + 1) / 2;
    static constexpr size_t off_masks = 0;
    static constexpr size_t sz_masks = (size_t)S::v * ST * 16;
    static constexpr size_t sz_mask2 = (size_t)QL * ST * 16, sz_upk = pad16((size_t)TRI * NQ * 4);
    static_assert(sz_mask2 + sz_upk <= sz_masks, "second-step masks and P3 fit");
    static constexpr size_t off_mask2 = 0, off_upk = sz_mask2;
    static constexpr size_t off_T = sz_masks;
    static constexpr size_t off_o = off_T + (size_t)J * CH * 32 * 16;
    static constexpr size_t off_ctr = off_o + pad16(S::o_bytes);
    static constexpr size_t total = off_ctr + 16;
};

// Rows r0 .. r0 + 3 of the upper-triangular P1, p1 bytes from base4; word q.
template <int SET>
struct TriRows {
    using S = Set<SET>;
    uint32_t p1, q4;
    int r0, row_l;
    __device__ __forceinline__ void start(uint32_t (&bit)[4], int c) const {
#pragma unroll
        for (int i = 0; i < 4; i++) bit[i] = 8u * (p1 + (uint32_t)(tri(min(r0 + i, S::v - 1), c, S::v) * S::menc) + q4);
    }
    __device__ __forceinline__ void next(uint32_t (&bit)[4], int) const {
#pragma unroll
        for (int i = 0; i < 4; i++) bit[i] += 8 * S::menc;
    }
    __device__ __forceinline__ void next_all(uint32_t (&bit)[4], int c) const { next(bit, c); }
    __device__ __forceinline__ bool keep(int i, int c) const { return c >= r0 + i; }
    __device__ __forceinline__ void ahead(const uint32_t *base4, int c) const { row_ahead(base4, p1, row_l, c); }
    __device__ static __forceinline__ void row_ahead(const uint32_t *base4, uint32_t p1, int r, int c) {
        if (r < S::v && c >= r && c < S::v)
            l2_prefetch(base4, p1 + (uint32_t)(tri(r, c, S::v) * S::menc), (uint32_t)(min(S::v - c, QUAD_AHEAD) * S::menc));
    }
};

// O[c][j] from the packed O in shared memory.
template <int SET>
__device__ __forceinline__ uint32_t o_nibble(const uint8_t *s_O, int c, int j) {
    const int q = c * Set<SET>::o + j;
    return (uint32_t)(s_O[q >> 1] >> ((q & 1) * 4)) & 0xFu;
}

// The quad of entries (r0 + i, j) of P2 (v x o), word q, as packed words (rows past v: any value).
template <int SET, bool RO>
__device__ __forceinline__ void p2_words(const uint32_t *base4, uint32_t p2, int r0, int j, int q, uint32_t (&w)[4]) {
    using S = Set<SET>;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint32_t bit = 8u * (p2 + (uint32_t)((min(r0 + i, S::v - 1) * S::o + j) * S::menc) + 4u * q);
        w[i] = raw_value(ld_raw<RO, true>(base4, bit, QuadCfg<SET>::bytes(q)), bit);
    }
}

// n (1..4) bytes of a packed word to any address.
__device__ __forceinline__ void store_word(uint8_t *p, uint32_t w, int n) {
    if (n == 4 && (reinterpret_cast<uintptr_t>(p) & 3) == 0) {
        *reinterpret_cast<uint32_t *>(p) = w;
    } else if ((reinterpret_cast<uintptr_t>(p) & 1) == 0 && (n & 1) == 0) {
        *reinterpret_cast<uint16_t *>(p) = (uint16_t)w;
        if (n == 4) *reinterpret_cast<uint16_t *>(p + 2) = (uint16_t)(w >> 16);
    } else {
#pragma unroll
        for (int b = 0; b < 4; b++)
            if (b < n) p[b] = (uint8_t)(w >> (8 * b));
    }
}

// P3 of one instance: P1 || P2 at P1, O (o_bytes) already in shared memory at off_o (of every CTA of a
// cluster); writes the packed upper triangle to P3out (rank 0).  All NT threads must call it.  RO:
// P1 and P2 are not written in this kernel.
template <int SET, int CL, bool RO, class C = KeyCfg<SET, CL>>
__device__ __forceinline__ void p3_instance(uint8_t *smem, int tid, const uint8_t *P1, uint8_t *P3out, int rank = 0) {
    using S = Set<SET>;
    constexpr int J = C::J, NQ = C::NQ, NT = C::NT, NP = C::NP, ULP = C::CH * 32;
    uint4 *masks = reinterpret_cast<uint4 *>(smem + C::off_masks);
    uint4 *mask2 = reinterpret_cast<uint4 *>(smem + C::off_mask2);
    uint32_t *upk = reinterpret_cast<uint32_t *>(smem + C::off_upk);  // [pair][NQ]
    uint4 *T = reinterpret_cast<uint4 *>(smem + C::off_T);            // [j][unit]
    const uint8_t *s_O = smem + C::off_o;
    int *s_next = reinterpret_cast<int *>(smem + C::off_ctr);
    const int warp = tid >> 5, lane = tid & 31;
    const uint32_t mis = (uint32_t)(reinterpret_cast<uintptr_t>(P1) & 3);
    const uint32_t *base4 = reinterpret_cast<const uint32_t *>(P1 - mis);
    if constexpr (CL == 1 && RO) {
        for (int r = tid; r < S::v; r += NT) TriRows<SET>::row_ahead(base4, mis, r, r);
        l2_prefetch_range(base4, mis + S::p1, S::p2, tid, NT);
    }
    auto scalar = [&](int c, int j) { return o_nibble<SET>(s_O, c, j); };
    auto quad_scalar = [&](int t, int i, int j) {
        const int c = 4 * (rank + t * NP) + i;
        return c < S::v ? scalar(c, j) : 0u;
    };
    if (tid == 0) *s_next = 0;
    build_masks9<J>(reinterpret_cast<uint32_t *>(masks), S::v, tid, NT, scalar);
    if constexpr (C::PC > 1) {
        for (int i = tid; i < J * ULP; i += NT) T[i] = make_uint4(0, 0, 0, 0);
    }
    __syncthreads();
    for (;;) {
        const int item = warp_next(s_next, lane);
        if (item >= C::CH * C::PC) break;
        const int chunk = item / C::PC, piece = item - chunk * C::PC;
        const int u = chunk * 32 + lane, t = u / NQ, q = u - t * NQ;
        const int r0 = 4 * (rank + t * NP);
        const int qmin = rank + (chunk * 32 / NQ) * NP, qmax = min(rank + ((chunk * 32 + 31) / NQ) * NP, C::QN - 1);
        const int c_lo = min(4 * qmin, S::v), len = S::v - c_lo;
        const int tl = chunk * 32 / NQ + (lane >> 2);
        QuadAcc<J> acc;
        acc.zero();
        const TriRows<SET> rows{mis, (uint32_t)(4 * q), r0,
                                RO && tl <= (chunk * 32 + 31) / NQ ? 4 * (rank + tl * NP) + (lane & 3) : S::v};
        quad_columns<SET, J, RO, C::D>(acc, rows, base4, QuadCfg<SET>::bytes(q), c_lo + len * piece / C::PC,
                                    c_lo + len * (piece + 1) / C::PC, 4 * qmax + 4, masks, mis == 0);
        const uint32_t rm = quad_row_mask(r0, S::v);
#pragma unroll
        for (int j = 0; j < J; j++) {
            G4 v = acc.fold(j);
            if (C::PC == 1 || piece == 0) {  // + P2[r][j]
                uint32_t w[4];
                p2_words<SET, RO>(base4, mis + S::p1, r0, j, q, w);
                v = g4_xor(v, quad_planes(w[0], w[1], w[2], w[3]));
            }
            v = g4_and(v, rm);
            if constexpr (C::PC > 1) g4_atomic_xor(T + j * ULP + u, v);
            else g4_st(T + j * ULP + u, v);
        }
    }
    __syncthreads();
    build_quad_masks9<J>(reinterpret_cast<uint32_t *>(mask2), C::QL, tid, NT, quad_scalar);
    for (int i = tid; i < C::TRI * NQ; i += NT) upk[i] = 0;
    __syncthreads();
    quad_pairs<SET, C>(T, ULP, mask2, upk, 0, warp, lane, [](int a, int b) { return tri(a, b, J); });
    __syncthreads();
    if constexpr (CL > 1) {
        cluster_barrier();
        if (rank == 0)
            for (int i = tid; i < C::TRI * NQ; i += NT) upk[i] = xor_cluster<CL>(upk + i);
        cluster_barrier();
        if (rank != 0) return;
        __syncthreads();
    }
    for (int i = tid; i < C::TRI * NQ; i += NT) {
        const int p = i / NQ, q = i - p * NQ;
        store_word(P3out + p * S::menc + 4 * q, upk[i], QuadCfg<SET>::bytes(q));
    }
}

// L = (P1 + P1^T) O + P2, in place over P2.
template <int SET, int CL_ = 1>
struct LCfg {
    using S = Set<SET>;
    static constexpr int CL = CL_, J = S::o, NQ = QuadCfg<SET>::NQ, ST = QuadAcc<J>::ST;
    static constexpr int QN = (S::v + 3) / 4, CH = (QN * NQ + 31) / 32;  // chunks, every one v columns long
    // expand-sk at 2,072 (us per instance): MAYO_1 0.410 with three CTAs per SM, 0.424 with four (128
    // registers); MAYO_2 0.327 with four warps, 0.344 with two; MAYO_3 0.901 with two CTAs of six warps,
    // 1.02 with eight warps, two columns ahead; MAYO_5 2.27 with eight warps, two ahead, 2.40 with
    // eleven, one ahead
    // With several CTAs per instance a chunk's columns are split over eight warps, whose sums meet in
    // shared memory: a lone warp ran a chunk's 78 to 142 columns one after another.  expand-sk for one
    // secret, MAYO_1 57 -> 38 us, MAYO_2 64 -> 45, MAYO_3 72 -> 50, MAYO_5 83 -> 74; at 72 secrets MAYO_1
    // 71 -> 64, MAYO_5 210 -> 212.
    static constexpr int CHC = (CH + CL - 1) / CL;  // chunks of a CTA
    static constexpr int CW = CL > 1 ? 8 : (SET == 1 ? 4 : SET == 2 ? 4 : SET == 3 ? 6 : 8);
    static constexpr int NT = 32 * CW;
    static constexpr int D = SET == 5 ? 2 : 1;  // columns loaded ahead
    static constexpr int MINB = CL > 1 ? 1 : (SET == 1 ? 3 : SET == 5 ? 1 : 2);
    static constexpr int PC = CL > 1 ? (2 * CW + CHC - 1) / CHC : 1;
    static constexpr size_t off_masks = 0;
    static constexpr size_t off_T = (size_t)S::v * ST * 16;
    static constexpr size_t off_o = off_T + (PC > 1 ? (size_t)J * CHC * 32 * 16 : 0);
    static constexpr size_t off_ctr = off_o + pad16(S::o_bytes);
    static constexpr size_t total = off_ctr + 16;
};

// Rows r0 .. r0 + 3 of P1 + P1^T without the diagonal: entry (r, c) is P1's (c, r) left of the
// diagonal.  lower: every row of the warp is there for all columns asked for (next_all's step).
template <int SET>
struct SymRows {
    using S = Set<SET>;
    uint32_t p1, q4;
    int r0;
    bool lower;
    __device__ __forceinline__ void start(uint32_t (&bit)[4], int c) const {
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int r = min(r0 + i, S::v - 1);
            bit[i] = 8u * (p1 + (uint32_t)((c < r ? tri(c, r, S::v) : tri(r, c, S::v)) * S::menc) + q4);
        }
    }
    // tri(c, r) - tri(c - 1, r) = v - c for c <= r
    __device__ __forceinline__ void next(uint32_t (&bit)[4], int c) const {
        const uint32_t lo = 8u * S::menc * (uint32_t)(S::v - c);
#pragma unroll
        for (int i = 0; i < 4; i++) bit[i] += c <= min(r0 + i, S::v - 1) ? lo : 8u * S::menc;
    }
    __device__ __forceinline__ void next_all(uint32_t (&bit)[4], int c) const {
        const uint32_t d = lower ? 8u * S::menc * (uint32_t)(S::v - c) : 8u * S::menc;
#pragma unroll
        for (int i = 0; i < 4; i++) bit[i] += d;
    }
    __device__ __forceinline__ bool keep(int i, int c) const { return c != r0 + i; }
    __device__ __forceinline__ void ahead(const uint32_t *, int) const {}
};

// L of one instance: P1 at P1 (then P2, which becomes L); O in shared memory at LCfg::off_o.
template <int SET, int CL>
__device__ __forceinline__ void l_instance(uint8_t *smem, int tid, const uint8_t *P1, uint8_t *P2, int rank) {
    using S = Set<SET>;
    using C = LCfg<SET, CL>;
    constexpr int J = C::J, NQ = C::NQ, NT = C::NT;
    uint4 *masks = reinterpret_cast<uint4 *>(smem + C::off_masks);
    const uint8_t *s_O = smem + C::off_o;
    int *s_next = reinterpret_cast<int *>(smem + C::off_ctr);
    const int lane = tid & 31;
    const uint32_t mis = (uint32_t)(reinterpret_cast<uintptr_t>(P1) & 3);
    const uint32_t *base4 = reinterpret_cast<const uint32_t *>(P1 - mis);
    uint4 *T = reinterpret_cast<uint4 *>(smem + C::off_T);  // [j][unit of this CTA]
    if (tid == 0) *s_next = 0;
    if constexpr (CL == 1) l2_prefetch_range(base4, mis, S::p1, tid, NT);  // read by rows and by columns
    build_masks9<J>(reinterpret_cast<uint32_t *>(masks), S::v, tid, NT,
                    [&](int c, int j) { return o_nibble<SET>(s_O, c, j); });
    if constexpr (C::PC > 1) {
        for (int i = tid; i < J * C::CHC * 32; i += NT) T[i] = make_uint4(0, 0, 0, 0);
    }
    __syncthreads();
    // words q of L[r0 + i][j] from the sum's planes
    auto store = [&](const G4 &f, int r0, int j, int q) {
        const G4 v = quad_planes(f.p0, f.p1, f.p2, f.p3);
        const uint32_t wd[4] = {v.p0, v.p1, v.p2, v.p3};
        uint32_t w[4];
        p2_words<SET, false>(base4, mis + S::p1, r0, j, q, w);
#pragma unroll
        for (int i = 0; i < 4; i++)
            if (r0 + i < S::v)
                store_word(P2 + (size_t)((r0 + i) * S::o + j) * S::menc + 4 * q, wd[i] ^ w[i], QuadCfg<SET>::bytes(q));
    };
    for (;;) {
        const int item = warp_next(s_next, lane), lc = C::PC > 1 ? item / C::PC : item, piece = item - lc * C::PC;
        const int chunk = rank + CL * lc;
        if (chunk >= C::CH) break;
        const int u = chunk * 32 + lane, t = u / NQ, q = u - t * NQ, r0 = 4 * t;
        const int qmin = chunk * 32 / NQ, qmax = min((chunk * 32 + 31) / NQ, C::QN - 1);
        QuadAcc<J> acc;
        acc.zero();
        SymRows<SET> rows{mis, (uint32_t)(4 * q), r0, false};
#pragma unroll 1
        for (int seg = 0; seg < 2; seg++) {  // from the diagonal on, then the columns left of every row
            rows.lower = seg == 1;
            int c0 = seg ? 0 : 4 * qmin, c1 = seg ? 4 * qmin : S::v;
            if constexpr (C::PC > 1) {  // the piece's columns
                c0 = max(c0, S::v * piece / C::PC);
                c1 = min(c1, S::v * (piece + 1) / C::PC);
            }
            quad_columns<SET, J, true, C::D>(acc, rows, base4, QuadCfg<SET>::bytes(q), c0, c1, seg ? 0 : 4 * qmax + 4, masks,
                                             mis == 0);
        }
        if constexpr (C::PC > 1) {
#pragma unroll
            for (int j = 0; j < J; j++) g4_atomic_xor(T + (j * C::CHC + lc) * 32 + lane, acc.fold(j));
        } else {
#pragma unroll
            for (int j = 0; j < J; j++) store(acc.fold(j), r0, j, q);
        }
    }
    if constexpr (C::PC > 1) {
        __syncthreads();
        for (int i = tid; i < J * C::CHC * 32; i += NT) {
            const int j = i / (C::CHC * 32), lu = i - j * (C::CHC * 32), chunk = rank + CL * (lu >> 5);
            const int u = chunk * 32 + (lu & 31), t = u / NQ, q = u - t * NQ;
            if (chunk < C::CH) store(g4_ld(T + i), 4 * t, j, q);
        }
    }
}

}  // namespace mayo
