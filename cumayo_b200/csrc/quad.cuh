// quad.cuh -- products of a per-instance key with a few vectors, the arithmetic behind every
// operation whose key is not shared by its batch:
//     T_j[r] = sum_c S[c][j] P[r][c]          (rows r of the key, columns c, vectors j)
//   keypair  P3 = Upper(O^T (P1 O + P2))      rows of P1, S = O           (src/keypair.cu:55-120)
//   expandsk L  = (P1 + P1^T) O + P2          rows of P1 + P1^T, S = O    (src/expandsk.cu:37-80)
//   sign     U = V^T P1 V, M = V L            rows of P1 and columns of L (src/sign.cu:256-330, 396-437)
//   verify   U = s^T P s                      rows of P1 | P2 and P3      (src/verify.cu:72-182)
//
// What bounds it: LOP3 issue (64 lanes per clock and SM).  The layout follows from that.
//   * Nine ANDs per product.  Multiplication in GF(16) has bilinear rank 9 over GF(2): with the nine
//     XOR forms f_d of an entry's four bit planes (Karatsuba on two levels) and the same forms m_d of
//     the scalar as all-ones / all-zero masks, s v is a fixed XOR of the nine words m_d & f_d.  A sum
//     of products accumulates A_d ^= m_d & f_d -- 9 LOP3 per 32 coordinates where the plane products
//     take 16 -- and recombines once per sum (forms_fold).
//   * A thread owns one unit -- four rows of the key (a quad) and one packed word (8 coordinates) --
//     and every vector j: 9 JB accumulators.  An entry is loaded, turned into planes (a 4x4 bit
//     transpose over the quad's four words: plane bit 4 e + i is coordinate e of row i) and into its
//     forms once, for all j; nothing of the key passes through shared memory and the column loop has
//     no barrier.  m-vectors of 39, 54 and 71 bytes fill 10, 14 and 18 words with no padding to 16.
//   * All lanes of a warp are at the same column, so the scalar masks ([column][j][d]) are 128-bit
//     shared-memory loads of one address per warp.  Such a load takes two clocks per SM, so the masks
//     (9 JB / 4 loads) and the key words (8 loads, two clocks each) keep the load pipe about as busy
//     as the products keep the logic pipe (MAYO_1: 62 and 57 clocks per column; measured 89).
// Verify at 3,552 / 3,552 / 2,072 / 1,036 instances with keys of their own (MAYO_1, 2, 3, 5): 0.33,
// 0.17, 0.66, 1.46 us per instance with the plane products (16 LOP3, rows staged
// in shared memory between barriers), 0.153, 0.064, 0.381, 0.752 here.
// Scalars enter only as masks and no address depends on them: constant time.
#pragma once

#include "common.cuh"

namespace mayo {

// XOR-accumulate a G4 into shared memory (atomic).
__device__ __forceinline__ void g4_atomic_xor(uint4 *dst, const G4 &g) {
    uint32_t *d = reinterpret_cast<uint32_t *>(dst);
    atomicXor(d + 0, g.p0);
    atomicXor(d + 1, g.p1);
    atomicXor(d + 2, g.p2);
    atomicXor(d + 3, g.p3);
}

// Named barrier over the first `n` threads (n a multiple of 32).
__device__ __forceinline__ void bar_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }

constexpr int NFORM = 9;

// The nine forms of four planes (or of the bits of a scalar, as masks).
__host__ __device__ __forceinline__ void forms_of(const G4 &v, uint32_t (&f)[NFORM]) {
    f[0] = v.p0;
    f[1] = v.p1;
    f[2] = v.p2;
    f[3] = v.p3;
    f[4] = v.p0 ^ v.p1;
    f[5] = v.p2 ^ v.p3;
    f[6] = v.p0 ^ v.p2;
    f[7] = v.p1 ^ v.p3;
    f[8] = f[4] ^ f[5];
}
// Planes of the product (or of a sum of products) from the nine accumulated ANDs: the Karatsuba
// recombination c_0 .. c_6 of two polynomials of degree 3, reduced with x^4 = x + 1.
__host__ __device__ __forceinline__ G4 forms_fold(const uint32_t *A) {
    const uint32_t a01 = A[0] ^ A[1], a23 = A[2] ^ A[3];
    const uint32_t c1 = A[4] ^ a01;
    const uint32_t c2 = lop_xor3(A[6], a01, A[2]);
    const uint32_t c3 = lop_xor3(lop_xor3(A[8], A[4], A[5]), lop_xor3(A[6], A[7], a01), a23);
    const uint32_t c4 = lop_xor3(A[7], a23, A[1]);
    const uint32_t c5 = A[5] ^ a23;
    return G4{A[0] ^ c4, lop_xor3(c1, c4, c5), lop_xor3(c2, c5, A[3]), c3 ^ A[3]};
}

// 4x4 bit transpose at every nibble position by bit selects.  two / four: 2 and 4; as values the
// compiler cannot fold (quad_columns passes constant-bank words) the left shifts are IMADs, off the
// pipe that LOP3, SHF and PRMT share.
__host__ __device__ __forceinline__ G4 quad_planes(uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3,
                                                   uint32_t two = 2, uint32_t four = 4) {
    constexpr uint32_t M2 = 0x33333333u, M1 = 0x55555555u;
    const uint32_t a0 = (w0 & M2) | ((w2 * four) & ~M2), a2 = ((w0 >> 2) & M2) | (w2 & ~M2);
    const uint32_t a1 = (w1 & M2) | ((w3 * four) & ~M2), a3 = ((w1 >> 2) & M2) | (w3 & ~M2);
    return G4{(a0 & M1) | ((a1 * two) & ~M1), ((a0 >> 1) & M1) | (a1 & ~M1), (a2 & M1) | ((a3 * two) & ~M1),
              ((a2 >> 1) & M1) | (a3 & ~M1)};
}
static __constant__ uint32_t c_quad_mul[2] = {2, 4};
// Sum over a quad's four rows of each coordinate, as a packed word (8 nibbles).
__host__ __device__ __forceinline__ uint32_t quad_row_sum(const G4 &v) {
    const uint32_t p[4] = {v.p0, v.p1, v.p2, v.p3};
    uint32_t r = 0;
#pragma unroll
    for (int b = 0; b < 4; b++) {
        uint32_t x = p[b] ^ (p[b] >> 1);
        x ^= x >> 2;
        r |= (x & 0x11111111u) << b;
    }
    return r;
}

// Nine masks of a scalar nibble.
__device__ __forceinline__ void nibble_forms(uint32_t s, uint32_t (&f)[NFORM]) {
    const uint4 m = scalar_masks(s);
    forms_of(G4{m.x, m.y, m.z, m.w}, f);
}
// Nine masks of a quad of scalars: bit 4 e + i of every form belongs to scalar i.
__device__ __forceinline__ void quad_forms(uint32_t s0, uint32_t s1, uint32_t s2, uint32_t s3, uint32_t (&f)[NFORM]) {
    const uint32_t q = s0 | (s1 << 4) | (s2 << 8) | (s3 << 12);
    uint32_t p[4];
#pragma unroll
    for (int b = 0; b < 4; b++) {
        const uint32_t x = q >> b;
        const uint32_t n = (x & 1u) | ((x >> 3) & 2u) | ((x >> 6) & 4u) | ((x >> 9) & 8u);
        p[b] = n * 0x11111111u;
    }
    forms_of(G4{p[0], p[1], p[2], p[3]}, f);
}

// One word (8 coordinates) of a packed m-vector at any byte address, given as a bit offset from a
// 4-byte aligned base: the aligned word that holds its first byte and the next one.  Bit offsets keep
// the address arithmetic at an add, a shift and an IMAD.WIDE, and are the funnel shift's amount
// (modulo 32) as they stand.  SAFE: the second word is read only where the n bytes reach it (n < 4
// in the last word of an m-vector); otherwise it may hold only bytes of the entry that follows, so
// the caller uses SAFE for the last entry of a buffer: quad_columns for the last column of its range,
// past which the entry that follows may lie in another buffer.
struct RawWord {
    uint32_t lo, hi;
};
template <bool RO>
__device__ __forceinline__ uint32_t ld_word(const uint32_t *p) {
    return RO ? __ldg(p) : __ldca(p);
}
// AL: every word is 4-byte aligned (whole words: n is 4).
template <bool RO, bool SAFE, bool AL = false>
__device__ __forceinline__ RawWord ld_raw(const uint32_t *base4, uint32_t bit, int n) {
    const uint32_t *p = base4 + (bit >> 5);
    RawWord r;
    r.lo = ld_word<RO>(p);
    r.hi = AL ? 0u : !SAFE || (int)((bit >> 3) & 3u) + n > 4 ? ld_word<RO>(p + 1) : 0u;
    return r;
}
template <bool AL = false>
__device__ __forceinline__ uint32_t raw_value(const RawWord &r, uint32_t bit) {
    return AL ? r.lo : __funnelshift_r(r.lo, r.hi, bit);
}

// Ask L2 for bytes [at, at + n) from base4 (n > 0), rounded out to 16-byte units, each of which
// holds a requested byte.
__device__ __forceinline__ void l2_prefetch(const uint32_t *base4, uint32_t at, uint32_t n) {
    const uint64_t a = reinterpret_cast<uint64_t>(base4) + at, b = (a + n + 15) & ~15ull, a0 = a & ~15ull;
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a0), "r"((uint32_t)(b - a0)) : "memory");
}

template <int SET>
struct QuadCfg {
    using S = Set<SET>;
    static constexpr int NQ = (S::menc + 3) / 4;             // words of an m-vector
    static constexpr int LAST = S::menc - 4 * (NQ - 1);      // bytes of the last one
    // coordinates of the last word (as a packed-word mask)
    static constexpr uint32_t LAST_MASK = S::m % 8 ? (1u << (4 * (S::m % 8))) - 1u : 0xFFFFFFFFu;
    __device__ static __forceinline__ int bytes(int q) { return q == NQ - 1 ? LAST : 4; }
};

// Accumulators of one unit for JB vectors.
template <int JB>
struct QuadAcc {
    static constexpr int NF = NFORM * JB;
    static constexpr int ST = (NF + 3) / 4;  // uint4 of masks per column
    uint32_t A[NF];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int i = 0; i < NF; i++) A[i] = 0;
    }
    // A[j][d] ^= mask[j][d] & f[d]
    __device__ __forceinline__ void madd(const uint4 *mp, const uint32_t (&f)[NFORM]) {
#pragma unroll
        for (int ch = 0; ch < ST; ch++) {
            const uint4 m = mp[ch];
            const uint32_t mm[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
            for (int e = 0; e < 4; e++)
                if (4 * ch + e < NF) A[4 * ch + e] = lop_xand(A[4 * ch + e], mm[e], f[(4 * ch + e) % NFORM]);
        }
    }
    __device__ __forceinline__ G4 fold(int j) const { return forms_fold(A + NFORM * j); }
};

// The same for a range of any length, by the threads of a CTA.
__device__ __forceinline__ void l2_prefetch_range(const uint32_t *base4, uint32_t at, uint32_t n, int tid, int nthreads) {
    constexpr uint32_t STEP = 2048;
    for (uint32_t o = STEP * (uint32_t)tid; o < n; o += STEP * (uint32_t)nthreads) l2_prefetch(base4, at + o, min(STEP, n - o));
}

// Columns [c0, c1) of one unit: acc += S[c] * (the quad's entries of column c).  `rows` gives the
// addresses: bit[4] (bit offsets from base4, the unit's word included), rows.start(bit, c) for
// column c, rows.next(bit, c) from column c - 1 to c (next_all: the same where c - 1 >= c_chk),
// rows.keep(i, c) whether row i has an entry in column c (asked for c < c_chk only; a row's offset is
// in bounds for every c), rows.ahead(base4, c) to ask L2 for the warp's rows from column c on.  The loads of column c + D are issued before the
// products of column c.  All lanes of a warp must pass the same c0, c1 and c_chk.
// Three loops, so that the long one (every row has an entry, no column is the last) has no tests.
constexpr int QUAD_AHEAD = 16;  // columns per L2 request
template <int SET, int JB, bool RO, int D, bool AL, class Rows>
__device__ __forceinline__ void quad_columns_t(QuadAcc<JB> &acc, const Rows &rows, const uint32_t *base4, int n, int c0,
                                             int c1, int c_chk, const uint4 *masks) {
    if (c0 >= c1) return;
    const uint32_t two = c_quad_mul[0], four = c_quad_mul[1];
    uint32_t bit[4], bl[4], w[4];  // offsets of the column in work and of the last one loaded
    RawWord raw[D][4];
    rows.start(bit, c0);
#pragma unroll
    for (int i = 0; i < 4; i++) bl[i] = bit[i];
#pragma unroll
    for (int d = 0; d < D; d++) {
        if (d > 0 && c0 + d < c1) rows.next(bl, c0 + d);
#pragma unroll
        for (int i = 0; i < 4; i++) raw[d][i] = ld_raw<RO, true, AL>(base4, bl[i], n);
    }
    const uint4 *mp = masks + (size_t)c0 * QuadAcc<JB>::ST;
    auto take = [&] {
#pragma unroll
        for (int i = 0; i < 4; i++) w[i] = raw_value<AL>(raw[0][i], bit[i]);
#pragma unroll
        for (int d = 0; d + 1 < D; d++)
#pragma unroll
            for (int i = 0; i < 4; i++) raw[d][i] = raw[d + 1][i];
    };
    auto load_last = [&] {  // column c + D, not the last of the range
#pragma unroll
        for (int i = 0; i < 4; i++) raw[D - 1][i] = ld_raw<RO, false, AL>(base4, bl[i], n);
    };
    auto products = [&] {
        uint32_t f[NFORM];
        forms_of(quad_planes(w[0], w[1], w[2], w[3], two, four), f);
        acc.madd(mp, f);
        mp += QuadAcc<JB>::ST;
    };
    int c = c0;
    const int e2 = c1 - 1 - D, e1 = min(c_chk, e2);
#pragma unroll 1
    while (c < e2) {
        rows.ahead(base4, c + QUAD_AHEAD);
        const int b1 = min(c + QUAD_AHEAD, e1), b2 = min(c + QUAD_AHEAD, e2);
#pragma unroll 1
        for (; c < b1; c++) {
            take();
#pragma unroll
            for (int i = 0; i < 4; i++) w[i] = rows.keep(i, c) ? w[i] : 0u;
            rows.next(bl, c + D);
            load_last();
            rows.next(bit, c + 1);
            products();
        }
#pragma unroll D
        for (; c < b2; c++) {
            take();
            rows.next_all(bl, c + D);
            load_last();
            rows.next_all(bit, c + 1);
            products();
        }
    }
#pragma unroll 1
    for (; c < c1; c++) {  // the last columns
        take();
#pragma unroll
        for (int i = 0; i < 4; i++) w[i] = c >= c_chk || rows.keep(i, c) ? w[i] : 0u;
        if (c + D < c1) {
            rows.next(bl, c + D);
#pragma unroll
            for (int i = 0; i < 4; i++) raw[D - 1][i] = ld_raw<RO, true, AL>(base4, bl[i], n);
        }
        rows.next(bit, c + 1);
        products();
    }
}

// m-vectors of whole words (MAYO_2: 32 bytes) from a 4-byte aligned key need one load per word and no
// shift.
template <int SET, int JB, bool RO, int D, class Rows>
__device__ __forceinline__ void quad_columns(QuadAcc<JB> &acc, const Rows &rows, const uint32_t *base4, int n, int c0,
                                             int c1, int c_chk, const uint4 *masks, bool aligned) {
    if (Set<SET>::menc % 4 == 0 && aligned)
        quad_columns_t<SET, JB, RO, D, Set<SET>::menc % 4 == 0>(acc, rows, base4, n, c0, c1, c_chk, masks);
    else
        quad_columns_t<SET, JB, RO, D, false>(acc, rows, base4, n, c0, c1, c_chk, masks);
}

// Rows r0 .. r0 + 3 of [[P1, P2], [0, P3]] (n x n), the matrix p bytes from base4; word q.  row_l:
// the row this lane asks L2 for (a row of one of the warp's quads, or >= n for none).
template <int SET>
struct PubRows {
    using S = Set<SET>;
    uint32_t p, q4;
    int r0, row_l;
    // entry index of (r, c), c >= r (a valid index for every c when r is a row of P1 or c >= v)
    __device__ static __forceinline__ int entry(int r, int c) {
        return c < S::v ? tri(r, c, S::v)
               : r < S::v ? S::e1 + r * S::o + (c - S::v)
                          : S::e1 + S::v * S::o + tri(r - S::v, c - S::v, S::o);
    }
    __device__ __forceinline__ void start(uint32_t (&bit)[4], int c) const {
#pragma unroll
        for (int i = 0; i < 4; i++) {
            int r = min(r0 + i, S::n - 1);
            if (c < S::v) r = min(r, S::v - 1);  // rows of P3 have no entry here: keep() drops them
            bit[i] = 8u * (p + (uint32_t)(entry(r, c) * S::menc) + q4);
        }
    }
    __device__ __forceinline__ void next(uint32_t (&bit)[4], int) const {  // not across column v
#pragma unroll
        for (int i = 0; i < 4; i++) bit[i] += 8 * S::menc;
    }
    __device__ __forceinline__ void next_all(uint32_t (&bit)[4], int c) const { next(bit, c); }
    __device__ __forceinline__ bool keep(int i, int c) const { return c >= r0 + i; }
    __device__ __forceinline__ void ahead(const uint32_t *base4, int c) const { row_ahead(base4, p, row_l, c); }
    // columns c .. c + QUAD_AHEAD - 1 of row r, up to the end of its run
    __device__ static __forceinline__ void row_ahead(const uint32_t *base4, uint32_t p, int r, int c) {
        if (r < S::n && c >= r && c < S::n) {
            const int end = c < S::v ? S::v : S::n, w = min(end - c, QUAD_AHEAD);
            l2_prefetch(base4, p + (uint32_t)(entry(r, c) * S::menc), (uint32_t)(w * S::menc));
        }
    }
};

// The next work item of a CTA's counter, for a whole warp (a uniform value).
__device__ __forceinline__ int warp_next(int *counter, int lane) {
    __syncwarp();
    return (int)__reduce_or_sync(0xffffffffu, lane == 0 ? (uint32_t)atomicAdd(counter, 1) : 0u);
}

// Which rows of a quad exist (r0 + i < nrows), as a plane mask.
__device__ __forceinline__ uint32_t quad_row_mask(int r0, int nrows) {
    uint32_t m = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) m |= r0 + i < nrows ? 0x11111111u << i : 0u;
    return m;
}
__device__ __forceinline__ G4 g4_and(const G4 &v, uint32_t m) { return G4{v.p0 & m, v.p1 & m, v.p2 & m, v.p3 & m}; }

// Masks [column][j][form] of nibble s(c, j), j < J, for columns [0, ncol): ST uint4 per column.
template <int J, class F>
__device__ __forceinline__ void build_masks9(uint32_t *masks, int ncol, int tid, int nthreads, F s) {
    constexpr int STW = QuadAcc<J>::ST * 4;
    for (int idx = tid; idx < ncol * J; idx += nthreads) {
        const int c = idx / J, j = idx - c * J;
        uint32_t f[NFORM];
        nibble_forms(s(c, j), f);
#pragma unroll
        for (int d = 0; d < NFORM; d++) masks[c * STW + j * NFORM + d] = f[d];
    }
}
// The same for quads t < nquads of scalars s(t, i, j), i < 4.
template <int J, class F>
__device__ __forceinline__ void build_quad_masks9(uint32_t *masks, int nquads, int tid, int nthreads, F s) {
    constexpr int STW = QuadAcc<J>::ST * 4;
    for (int idx = tid; idx < nquads * J; idx += nthreads) {
        const int t = idx / J, j = idx - t * J;
        uint32_t f[NFORM];
        quad_forms(s(t, 0, j), s(t, 1, j), s(t, 2, j), s(t, 3, j), f);
#pragma unroll
        for (int d = 0; d < NFORM; d++) masks[t * STW + j * NFORM + d] = f[d];
    }
}

// Barrier over the CTAs of a cluster (release / acquire of shared memory), and a word of the shared
// memory of CTA `rank` at this CTA's address p.
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t ld_cluster(const uint32_t *p, int rank) {
    uint32_t a = (uint32_t)__cvta_generic_to_shared(p), v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(a), "r"(rank));
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}

// XOR of the word at p over the CL CTAs of a cluster.
template <int CL>
__device__ __forceinline__ uint32_t xor_cluster(const uint32_t *p) {
    uint32_t v = *p;
#pragma unroll
    for (int r = 1; r < CL; r++) v ^= ld_cluster(p, r);
    return v;
}

// Exponent l of pair (a <= b) in y = sum z^l U_ab (src/verify.cu:185-211): pairs (0, k-1), (0, k-2), ...
__device__ __forceinline__ int pair_ell(int a, int b, int k) { return a * k - (a * (a - 1)) / 2 + (k - 1 - b); }

// The second step: X_ij = sum_r S[r][i] T_j[r] over the quads t0 <= t < C::QL of T ([j][ulp units]),
// packed and added to out[index(i <= j)][NQ].  A unit is (j, word); masks2: the quads' scalars.
template <int SET, class C, class F>
__device__ __forceinline__ void quad_pairs(const uint4 *T, int ulp, const uint4 *mask2, uint32_t *out, int t0, int warp,
                                           int lane, F index) {
    constexpr int J = C::J, NQ = C::NQ;
#pragma unroll 1
    for (int task = warp; task < C::CH2 * C::P2; task += C::CW) {
        const int ch = task / C::P2, pc = task - ch * C::P2;
        const int u = ch * 32 + lane, uc = min(u, J * NQ - 1), j = uc / NQ, q = uc - j * NQ;
        QuadAcc<J> acc;
        acc.zero();
        const uint4 *Tj = T + j * ulp + q;
#pragma unroll 1
        for (int t = max(C::QL * pc / C::P2, t0); t < C::QL * (pc + 1) / C::P2; t++) {
            uint32_t f[NFORM];
            forms_of(g4_ld(Tj + t * NQ), f);
            acc.madd(mask2 + t * C::ST, f);
        }
        if (u < J * NQ) {
            const uint32_t lm = q == NQ - 1 ? QuadCfg<SET>::LAST_MASK : 0xFFFFFFFFu;
#pragma unroll
            for (int i = 0; i < J; i++)
                atomicXor(out + index(min(i, j), max(i, j)) * NQ + q, quad_row_sum(acc.fold(i)) & lm);
        }
    }
}

// y = sum_l z^l U_l mod f(z) for packed U_l (upk[l][NQ]) by warps 0 .. nwarps - 1 (all their threads),
// in place of a Horner chain over the pairs: word x of the unreduced sum (lane x) collects every U_l
// shifted by l coordinates, the warps take every nwarps-th l and combine by XOR in yext (32 words,
// zeroed by the caller); y_fold then reduces it once (pairs + 3 < m).
template <int SET>
__device__ __forceinline__ void y_accumulate(const uint32_t *upk, uint32_t *yext, int warp, int nwarps, int lane) {
    using S = Set<SET>;
    constexpr int NQ = QuadCfg<SET>::NQ;
    static_assert(NQ + (S::pairs + 6) / 8 + 1 <= 32, "one lane per word");
    uint32_t y = 0;
#pragma unroll 1
    for (int l = warp; l < S::pairs; l += nwarps) {
        const int qa = lane - (l >> 3);
        const uint32_t hi = qa >= 0 && qa < NQ ? upk[l * NQ + qa] : 0u;
        const uint32_t lo = qa >= 1 && qa <= NQ ? upk[l * NQ + qa - 1] : 0u;
        y ^= __funnelshift_l(lo, hi, 4 * (l & 7));
    }
    if (y) atomicXor(yext + lane, y);
}
// Word `lane` of y (0 past the m-vector) from the unreduced sum; one warp.
template <int SET>
__device__ __forceinline__ uint32_t y_fold(const uint32_t *yext, int lane) {
    using S = Set<SET>;
    constexpr int NQ = QuadCfg<SET>::NQ;
    const uint32_t own = yext[lane];
    // coordinates m .. of the sum, moved to 0 ..
    constexpr int Q = S::m / 8, sh = 4 * (S::m % 8);
    const uint32_t a = lane + Q < 32 ? yext[(lane + Q) & 31] : 0u, b = lane + Q + 1 < 32 ? yext[(lane + Q + 1) & 31] : 0u;
    const uint32_t h = __funnelshift_r(a, b, sh);
    uint32_t y = lane < NQ ? (lane == NQ - 1 ? own & QuadCfg<SET>::LAST_MASK : own) : 0u;
#pragma unroll
    for (int n = 0; n < 4; n++) {
        if (S::cf(n) == 0) continue;
        const uint32_t mc = nib8_mul_const(h, S::cf(n));
        uint32_t prev = __shfl_up_sync(0xffffffffu, mc, 1);
        if (lane == 0) prev = 0;
        y ^= n ? (mc << (4 * n)) | (prev >> ((32 - 4 * n) & 31)) : mc;
    }
    return lane < NQ ? y : 0u;
}

}  // namespace mayo
