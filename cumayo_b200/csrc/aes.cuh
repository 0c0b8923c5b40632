// aes.cuh -- AES-128 in the counter mode the reference uses for P1||P2 expansion
// (reference src/aes128_ctr.cu:124-283): key = seed_pk, block i encrypts the 16-byte counter
// 0^8 || BE64(i), output bytes in standard AES order, a final partial block keeps its leading
// bytes.
//
// B200 layout: the round table T0 (Te0 of FIPS-197 in big-endian words) replicated 32 times in
// shared memory, entry x of copy c at word 32*x + c, so lane c always hits bank c and the 16
// data-dependent lookups of a round never conflict.  The other three round tables are byte
// rotations of T0.  The expansion kernel keeps all four (128 KB, one persistent CTA per SM); the
// work-queue kernel's keypair keeps as many as fit in the area its P3 uses next and rotates with PRMT
// for the others.  The S-box for the last round is byte 1 of T0[x].  Tables are computed at compile time from GF(2^8) arithmetic.
#pragma once

#include <type_traits>

#include "common.cuh"

namespace mayo {

struct AesTables {
    uint32_t te0[256];
    uint8_t sbox[256];
};

__host__ __device__ constexpr uint8_t gf256_mulc(uint8_t a, uint8_t b) {
    uint8_t r = 0;
    for (int i = 0; i < 8; i++) {
        if (b & 1) r ^= a;
        uint8_t hi = a & 0x80;
        a = (uint8_t)(a << 1);
        if (hi) a ^= 0x1B;
        b >>= 1;
    }
    return r;
}

__host__ __device__ constexpr AesTables make_aes_tables() {
    AesTables t{};
    // exp/log over the generator 0x03
    uint8_t ex[256] = {}, lg[256] = {};
    uint8_t g = 1;
    for (int i = 0; i < 255; i++) {
        ex[i] = g;
        lg[g] = (uint8_t)i;
        g = gf256_mulc(g, 3);
    }
    for (int x = 0; x < 256; x++) {
        uint8_t inv = x ? ex[(255 - lg[x]) % 255] : 0;
        uint8_t s = inv, r = inv;
        for (int i = 0; i < 4; i++) {
            r = (uint8_t)((r << 1) | (r >> 7));
            s ^= r;
        }
        s ^= 0x63;
        t.sbox[x] = s;
        t.te0[x] = ((uint32_t)gf256_mulc(s, 2) << 24) | ((uint32_t)s << 16) | ((uint32_t)s << 8) |
                   (uint32_t)gf256_mulc(s, 3);
    }
    return t;
}

__constant__ AesTables c_aes = make_aes_tables();

__device__ __forceinline__ uint32_t ror8(uint32_t x) { return __byte_perm(x, x, 0x0321); }
__device__ __forceinline__ uint32_t ror16(uint32_t x) { return __byte_perm(x, x, 0x1032); }
__device__ __forceinline__ uint32_t ror24(uint32_t x) { return __byte_perm(x, x, 0x2103); }
__device__ __forceinline__ uint32_t byte_of(uint32_t x, int b) { return __byte_perm(x, 0, 0x4440 | b); }

// AES-128 key schedule (FIPS-197 5.2) from 16 key bytes at any address; `sb` is the S-box (the
// constant-memory copy by default, a shared-memory copy where threads look up different bytes).
__device__ inline void aes128_key_schedule(const uint8_t *key, uint32_t *rk, const uint8_t *sb = nullptr) {
    if (!sb) sb = c_aes.sbox;
#pragma unroll
    for (int i = 0; i < 4; i++)
        rk[i] = ((uint32_t)key[4 * i] << 24) | ((uint32_t)key[4 * i + 1] << 16) | ((uint32_t)key[4 * i + 2] << 8) |
                key[4 * i + 3];
    uint32_t rcon = 1;
#pragma unroll
    for (int i = 4; i < 44; i++) {
        uint32_t t = rk[i - 1];
        if (i % 4 == 0) {
            t = (t << 8) | (t >> 24);
            t = ((uint32_t)sb[t >> 24] << 24) | ((uint32_t)sb[(t >> 16) & 0xFF] << 16) |
                ((uint32_t)sb[(t >> 8) & 0xFF] << 8) | sb[t & 0xFF];
            t ^= rcon << 24;
            rcon = gf256_mulc((uint8_t)rcon, 2);
        }
        rk[i] = rk[i - 4] ^ t;
    }
}

// The four big-endian state words of an encrypted counter block.
struct AesOut {
    uint32_t w0, w1, w2, w3;
};

// The table stride (128 bytes) as a value the compiler cannot fold, for kernels without a
// launch argument for it: a constant-bank operand keeps the address arithmetic an IMAD.
__constant__ uint32_t c_aes_stride = 128;

// NTAB replicated round tables in shared memory, 32 KB apart from `base` (the shared-memory address
// of T0 with this lane's column added):
//   NTAB = 4: T0, ror8(T0), ror16(T0), ror24(T0)   (the expansion kernel, 128 KB)
//   NTAB = 3: T0, ror8(T0), ror16(T0)   (the work queue's keypair, as many as its P3 area holds)
//   NTAB = 2: T0, ror16(T0)
//   NTAB = 1: T0
// the other round tables by PRMT rotations.  A lookup is a byte extraction, one IMAD for the
// address (the multiplier `k128` = 128 is a kernel argument or a constant-bank value, so the
// address arithmetic stays on the IMAD pipe instead of joining the extractions, rotations and
// XORs on the logic pipe, which with the table reads sets the pace) and the read.  Measured at
// MAYO_1's 1,024 x 9,031 blocks, all rounds by lookups: one table 0.234 ms, two 0.222, three (two CTAs
// of 384 threads per SM) 0.203; with the first two rounds shared (AesRun), persistent CTAs: three
// 0.197, four and a preparing warp 0.174.  133 lookups of a block at one wavefront each take 0.137.
template <int NTAB>
struct AesLut {
    static_assert(NTAB >= 1 && NTAB <= 4, "one to four tables");
    uint32_t base, k128;
    template <int T>
    __device__ __forceinline__ uint32_t ld(uint32_t x) const {
        uint32_t v;
        if constexpr (T == 0)
            asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(x * k128 + base));
        else if constexpr (T == 1)
            asm volatile("ld.shared.u32 %0, [%1+32768];" : "=r"(v) : "r"(x * k128 + base));
        else if constexpr (T == 2)
            asm volatile("ld.shared.u32 %0, [%1+65536];" : "=r"(v) : "r"(x * k128 + base));
        else
            asm volatile("ld.shared.u32 %0, [%1+98304];" : "=r"(v) : "r"(x * k128 + base));
        return v;
    }
    __device__ __forceinline__ uint32_t r0(uint32_t x) const { return ld<0>(x); }  // T0[x]
    __device__ __forceinline__ uint32_t r8(uint32_t x) const {                      // ror8(T0[x])
        if constexpr (NTAB >= 3) return ld<1>(x);
        else return ror8(ld<0>(x));
    }
    __device__ __forceinline__ uint32_t r16(uint32_t x) const {  // ror16(T0[x])
        if constexpr (NTAB >= 3) return ld<2>(x);
        else if constexpr (NTAB == 2) return ld<1>(x);
        else return ror16(ld<0>(x));
    }
    __device__ __forceinline__ uint32_t r24(uint32_t x) const {  // ror24(T0[x])
        if constexpr (NTAB == 4) return ld<3>(x);
        else if constexpr (NTAB == 1) return ror24(ld<0>(x));
        else return ror8(r16(x));
    }
    // one output word of a round (without its round key)
    __device__ __forceinline__ uint32_t mix(uint32_t a, uint32_t b, uint32_t c, uint32_t d) const {
        return r0(a >> 24) ^ r8(byte_of(b, 2)) ^ r16(byte_of(c, 1)) ^ r24(byte_of(d, 0));
    }
    // the same of the last round: S-box = byte 1 of T0[x]
    __device__ __forceinline__ uint32_t last(uint32_t a, uint32_t b, uint32_t c, uint32_t d) const {
        return __byte_perm(__byte_perm(r0(a >> 24), r0(byte_of(b, 2)), 0x1500),
                           __byte_perm(r0(byte_of(c, 1)), r0(byte_of(d, 0)), 0x0015), 0x3254);
    }
};

// What the first two rounds of 256 consecutive counter blocks share (blk >> 8 the same).  Only byte 15
// of the input differs between them, so of round 1 only output word a changes, by one lookup, and of
// round 2 each output word by the one lookup that takes a byte of a: five lookups instead of 32.
struct AesRun {
    uint32_t ka, kb, kc, kd;  // round 2 without the bytes of a
};
// rk: the round keys (rk[0 .. 11] are read).  a0: word a of round 1 without byte 15's lookup, the same
// for every run of a key.
template <int NTAB, class RK>
__device__ __forceinline__ uint32_t aes_run_a0(const AesLut<NTAB> &t, const RK &rk) {
    return t.r0(rk[0] >> 24) ^ t.r8(byte_of(rk[1], 2)) ^ t.r16(byte_of(rk[2], 1)) ^ rk[4];
}
template <int NTAB, class RK>
__device__ __forceinline__ AesRun aes_run(const AesLut<NTAB> &t, const RK &rk, uint32_t blk_hi) {
    const uint32_t s0 = rk[0], s1 = rk[1], s2 = rk[2], s3 = (blk_hi << 8) ^ rk[3];
    const uint32_t b = t.mix(s1, s2, s3, s0) ^ rk[5], c = t.mix(s2, s3, s0, s1) ^ rk[6], d = t.mix(s3, s0, s1, s2) ^ rk[7];
    AesRun r;
    r.ka = t.r8(byte_of(b, 2)) ^ t.r16(byte_of(c, 1)) ^ t.r24(byte_of(d, 0)) ^ rk[8];
    r.kb = t.r0(b >> 24) ^ t.r8(byte_of(c, 2)) ^ t.r16(byte_of(d, 1)) ^ rk[9];
    r.kc = t.r0(c >> 24) ^ t.r8(byte_of(d, 2)) ^ t.r24(byte_of(b, 0)) ^ rk[10];
    r.kd = t.r0(d >> 24) ^ t.r16(byte_of(b, 1)) ^ t.r24(byte_of(c, 0)) ^ rk[11];
    return r;
}

// Encrypt N counter blocks side by side, block blk[i] of run run[i] (i < N): k3 = the low byte of rk[3],
// rk[i] = round key word 12 + i.
template <int NTAB, int N, class RK>
__device__ __forceinline__ void aes128_ctr_blocks(const AesLut<NTAB> &t, uint32_t a0, uint32_t k3, const AesRun (&run)[N],
                                                  const RK &rk, const uint32_t (&blk)[N], AesOut (&o)[N]) {
    uint32_t s[N][4];
#pragma unroll
    for (int i = 0; i < N; i++) {
        const uint32_t a1 = a0 ^ t.r24(byte_of(blk[i] ^ k3, 0));
        s[i][0] = run[i].ka ^ t.r0(a1 >> 24);
        s[i][1] = run[i].kb ^ t.r24(byte_of(a1, 0));
        s[i][2] = run[i].kc ^ t.r16(byte_of(a1, 1));
        s[i][3] = run[i].kd ^ t.r8(byte_of(a1, 2));
    }
#pragma unroll
    for (int r = 0; r < 7; r++) {  // rounds 3 .. 9
#pragma unroll
        for (int i = 0; i < N; i++) {
            const uint32_t a = t.mix(s[i][0], s[i][1], s[i][2], s[i][3]) ^ rk[4 * r];
            const uint32_t b = t.mix(s[i][1], s[i][2], s[i][3], s[i][0]) ^ rk[4 * r + 1];
            const uint32_t c = t.mix(s[i][2], s[i][3], s[i][0], s[i][1]) ^ rk[4 * r + 2];
            const uint32_t d = t.mix(s[i][3], s[i][0], s[i][1], s[i][2]) ^ rk[4 * r + 3];
            s[i][0] = a;
            s[i][1] = b;
            s[i][2] = c;
            s[i][3] = d;
        }
    }
#pragma unroll
    for (int i = 0; i < N; i++) {
        o[i].w0 = t.last(s[i][0], s[i][1], s[i][2], s[i][3]) ^ rk[28];
        o[i].w1 = t.last(s[i][1], s[i][2], s[i][3], s[i][0]) ^ rk[29];
        o[i].w2 = t.last(s[i][2], s[i][3], s[i][0], s[i][1]) ^ rk[30];
        o[i].w3 = t.last(s[i][3], s[i][0], s[i][1], s[i][2]) ^ rk[31];
    }
}

// Big-endian words -> little-endian words of the byte stream.
__device__ __forceinline__ uint32_t bswap32(uint32_t x) { return __byte_perm(x, 0, 0x0123); }

// Store 16 stream bytes (as 4 LE words) at any address, widest aligned stores possible.
__device__ __forceinline__ void st16(uint8_t *p, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    uintptr_t ad = reinterpret_cast<uintptr_t>(p);
    if ((ad & 15) == 0) {
        *reinterpret_cast<uint4 *>(p) = make_uint4(a, b, c, d);
    } else if ((ad & 7) == 0) {
        reinterpret_cast<uint2 *>(p)[0] = make_uint2(a, b);
        reinterpret_cast<uint2 *>(p)[1] = make_uint2(c, d);
    } else if ((ad & 3) == 0) {
        uint32_t *q = reinterpret_cast<uint32_t *>(p);
        q[0] = a;
        q[1] = b;
        q[2] = c;
        q[3] = d;
    } else {
        const uint32_t w[4] = {a, b, c, d};
#pragma unroll
        for (int i = 0; i < 16; i++) p[i] = (uint8_t)(w[i >> 2] >> (8 * (i & 3)));
    }
}

// Counter block blk's 16 stream bytes.
__device__ __forceinline__ void aes_store(uint8_t *out, uint32_t blk, const AesOut &o) {
    st16(out + (size_t)blk * 16, bswap32(o.w0), bswap32(o.w1), bswap32(o.w2), bswap32(o.w3));
}

// ---------------------------------------------------------------------------------------------
// Kernel: AES-CTR keystream of nbytes into a pitched pool.  An item is (instance, chunk): chunk x of an
// instance takes blocks [x * bpc, (x + 1) * bpc) to row + out_off, keyed by 16 bytes at row + key_off
// (or derived, see AesDerive).  A CTA builds the tables once and takes items blockIdx.x, + gridDim.x,
// ...; while its worker warps run one item, the last warp prepares the next one (key schedule, the
// chunk's AesRuns).  The workers take the item's blocks 64 at a time from a counter (32 where an item
// has few).  When the key overlaps the output (expand-pk, and expand-sk that does not derive, keep
// seed_pk in the last 16 output bytes until expansion), nbytes ends before the blocks that overlap the key and aes_ctr_tail_kernel finishes them afterwards, one
// thread per instance.
// ---------------------------------------------------------------------------------------------
constexpr int AES_WORKERS = 768, AES_THREADS = AES_WORKERS + 32;  // and the warp that prepares
constexpr int AES_BLOCKS_PER_ITEM = 53248;  // at most (a MAYO_5 key has 52,616)
constexpr int AES_ITEM_COST = 700;          // what an item costs besides its blocks, in blocks (its workers drain)
// What the tail kernel costs, in blocks: its launch and the one (MAYO_2) or two it takes one after the
// other.  Expand-pk of 32 / 40 / 48 MAYO_2, one item per key and no tail 26.7 us, split with the tail
// 22.2, 23.3, 25.4; of 48 / 52 MAYO_1 split 31.1, one item 34.
constexpr int AES_TAIL_COST = 2500, AES_TAIL_BLOCK_COST = 1250;
constexpr int AES_RUNS = AES_BLOCKS_PER_ITEM / 256 + 2;
constexpr size_t AES_SMEM = 4 * 256 * 32 * 4;  // T0 and its rotations by 8, 16, 24, each replicated 32 times

// Where an item's key comes from when the kernel derives it from the secret seed (DERIVE, the
// smallest batches): seed_pk || O = SHAKE256(seed_sk), seed_sk at the row's start, or first
// SHAKE128(LE64(rand_index + 2 inst + 1)) where `counter` is set (src/keypair.cu:35-50).  The preparing
// warp then also writes what the hash kernels would: O to row + o_off and, where key_off is used,
// seed_pk to row + key_off, for an instance's first chunk, while the workers are at it.
struct AesDerive {
    uint32_t sk_bytes, o_bytes, write_key, counter;
    size_t o_off;
    uint64_t rand_index;
};

template <bool DERIVE>
__global__ void __launch_bounds__(AES_THREADS, 1)
    aes_ctr_kernel(uint8_t *pool, size_t pitch, size_t key_off, size_t out_off, uint32_t nbytes, uint32_t bpc,
                   uint32_t chunks, uint32_t items, uint32_t k128, const AesDerive dv) {
    extern __shared__ uint32_t aes_smem[];  // [4][256 * 32] words
    __shared__ uint32_t s_rk[2][44];
    __shared__ uint4 s_run[2][AES_RUNS];
    __shared__ uint32_t s_a0[2];
    __shared__ int s_next[2];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < 256 * 32; i += AES_THREADS) {
        const uint32_t v = c_aes.te0[i >> 5];
        aes_smem[i] = v;
        aes_smem[256 * 32 + i] = ror8(v);
        aes_smem[2 * 256 * 32 + i] = ror16(v);
        aes_smem[3 * 256 * 32 + i] = ror24(v);
    }
    __syncthreads();
    const AesLut<4> lut{(uint32_t)__cvta_generic_to_shared(aes_smem + lane), k128};
    [[maybe_unused]] WarpKeccak wk;
    if constexpr (DERIVE) wk.setup(lane);
    // the last warp; returns its sponge state after the first block of seed_pk || O
    auto prepare = [&](int buf, uint32_t item) {
        const uint32_t inst = item / chunks, chunk = item - inst * chunks, b0 = chunk * bpc;
        uint8_t *row = pool + (size_t)inst * pitch;
        const uint8_t *key = row + key_off;
        uint64_t a = 0;
        if constexpr (DERIVE) {
            __shared__ uint64_t s_sk[8], s_key[2];  // the counter and the seed; seed_pk
            const uint8_t *sk = row;
            if (dv.counter) {
                if (lane == 0) s_sk[0] = dv.rand_index + (uint64_t)(uint32_t)(2u * inst) + 1;
                __syncwarp();
                uint8_t *seed = reinterpret_cast<uint8_t *>(s_sk + 1);
                warp_shake<168>(seed, (int)dv.sk_bytes, reinterpret_cast<const uint8_t *>(s_sk), 8, wk, lane);
                for (int i0 = 0; i0 < (int)dv.sk_bytes; i0 += 32) {
                    if (chunk == 0 && i0 + lane < (int)dv.sk_bytes) row[i0 + lane] = seed[i0 + lane];
                    __syncwarp();
                }
                sk = seed;
            }
            const int n = (int)dv.sk_bytes - 8 * lane;  // one block: sk_bytes < 136
            if (n > 0) a = ld_bytes(sk + 8 * lane, n < 8 ? n : 8);
            if (n >= 0 && n < 8) a ^= (uint64_t)0x1F << (8 * n);
            if (lane == 16) a ^= 0x8000000000000000ull;
            a = wk.permute(lane < 25 ? a : 0, lane);
            if (lane < 2) s_key[lane] = a;
            __syncwarp();
            key = reinterpret_cast<const uint8_t *>(s_key);
        }
        if (lane == 0) {
            aes128_key_schedule(key, s_rk[buf]);
            s_next[buf] = 0;
        }
        __syncwarp();
        const uint32_t *rk = s_rk[buf];
        const uint32_t runs = ((b0 & 255u) + bpc + 255u) / 256u;
        for (uint32_t h0 = 0; h0 < runs; h0 += 32) {
            const uint32_t h = h0 + (uint32_t)lane;
            if (h < runs) {
                const AesRun r = aes_run(lut, rk, (b0 >> 8) + h);
                s_run[buf][h] = make_uint4(r.ka, r.kb, r.kc, r.kd);
            }
            __syncwarp();
        }
        if (lane == 0) s_a0[buf] = aes_run_a0(lut, rk);
        return a;
    };
    // seed_pk and O of an instance from the state `a` (an instance's first chunk)
    auto squeeze = [&](uint32_t item, uint64_t a) {
        const uint32_t inst = item / chunks;
        if (item != inst * chunks) return;
        uint8_t *row = pool + (size_t)inst * pitch;
        const int total = 16 + (int)dv.o_bytes;
        for (int o = 0; o < total; o += 136) {
            if (o) a = wk.permute(a, lane);
            if (lane < 17) {
#pragma unroll
                for (int b = 0; b < 8; b++) {
                    const int at = o + 8 * lane + b;
                    const uint8_t v = (uint8_t)(a >> (8 * b));
                    if (at < 16) {
                        if (dv.write_key) row[key_off + at] = v;
                    } else if (at < total) {
                        row[dv.o_off + at - 16] = v;
                    }
                }
            }
            __syncwarp();
        }
    };
    constexpr int PREP = AES_WORKERS / 32;
    uint64_t state = 0;
    if (warp == PREP) state = prepare(0, blockIdx.x);  // gridDim.x <= items
    __syncthreads();
    const uint32_t grab = bpc < 2 * AES_WORKERS ? 32u : 64u, nblk = (nbytes + 15) / 16;
    int buf = 0;
#pragma unroll 1
    for (uint32_t item = blockIdx.x; item < items; item += gridDim.x, buf ^= 1) {
        if (warp == PREP) {
            const uint64_t a = state;
            if (item + gridDim.x < items) state = prepare(buf ^ 1, item + gridDim.x);
            if constexpr (DERIVE) squeeze(item, a);
            __syncthreads();
            continue;
        }
        uint32_t rk[32];
#pragma unroll
        for (int i = 0; i < 32; i++) rk[i] = s_rk[buf][12 + i];
        const uint32_t a0 = s_a0[buf], k3 = s_rk[buf][3];
        const uint32_t inst = item / chunks, b0 = (item - inst * chunks) * bpc, b1 = min(b0 + bpc, nblk);
        uint8_t *out = pool + (size_t)inst * pitch + out_off;
        for (;;) {
            uint32_t g = 0;
            if (lane == 0) g = (uint32_t)atomicAdd(&s_next[buf], (int)grab);
            g = b0 + __shfl_sync(0xffffffffu, g, 0);
            if (g >= b1) break;
#pragma unroll 1
            for (uint32_t blk = g + lane; blk < min(g + grab, b1); blk += 32) {
                const uint4 r = s_run[buf][(blk >> 8) - (b0 >> 8)];
                const AesRun run[1] = {{r.x, r.y, r.z, r.w}};
                const uint32_t n[1] = {blk};
                AesOut o[1];
                aes128_ctr_blocks(lut, a0, k3, run, rk, n, o);
                if (16 * blk + 16 <= nbytes) {
                    aes_store(out, blk, o[0]);
                } else {  // a last partial block keeps its leading bytes
                    const uint32_t w[4] = {bswap32(o[0].w0), bswap32(o[0].w1), bswap32(o[0].w2), bswap32(o[0].w3)};
#pragma unroll
                    for (uint32_t i = 0; i < 16; i++)
                        if (16 * blk + i < nbytes) out[(size_t)blk * 16 + i] = (uint8_t)(w[i >> 2] >> (8 * (i & 3)));
                }
            }
        }
        __syncthreads();
    }
}

// Blocks [nblk_main, ceil(nbytes/16)) for each instance (key read before any byte is written).
// One thread per instance, at most two blocks each; the threads of a warp look up different
// bytes, so the tables are copied to shared memory first (constant memory would serialise them).
constexpr int AES_TAIL_THREADS = 128;
static __global__ void __launch_bounds__(AES_TAIL_THREADS)
    aes_ctr_tail_kernel(uint8_t *pool, size_t pitch, size_t key_off, size_t out_off, uint32_t nblk_main,
                        uint32_t nbytes, uint32_t batch) {
    __shared__ uint32_t te[256];
    __shared__ uint8_t sb[256];
    for (int i = threadIdx.x; i < 256; i += AES_TAIL_THREADS) {
        te[i] = c_aes.te0[i];
        sb[i] = c_aes.sbox[i];
    }
    __syncthreads();
    const uint32_t inst = blockIdx.x * blockDim.x + threadIdx.x;
    if (inst >= batch) return;
    uint8_t *row = pool + (size_t)inst * pitch;
    uint32_t rk[44];
    aes128_key_schedule(row + key_off, rk, sb);
    const uint32_t nblk = (nbytes + 15) / 16;
    uint8_t buf[32];
    for (uint32_t blk = nblk_main; blk < nblk; blk++) {
        uint32_t s0 = rk[0], s1 = rk[1], s2 = rk[2], s3 = blk ^ rk[3];
        for (int r = 1; r < 10; r++) {
            const uint32_t t0 = te[s0 >> 24] ^ ror8(te[(s1 >> 16) & 255]) ^ ror16(te[(s2 >> 8) & 255]) ^
                                ror24(te[s3 & 255]) ^ rk[4 * r];
            const uint32_t t1 = te[s1 >> 24] ^ ror8(te[(s2 >> 16) & 255]) ^ ror16(te[(s3 >> 8) & 255]) ^
                                ror24(te[s0 & 255]) ^ rk[4 * r + 1];
            const uint32_t t2 = te[s2 >> 24] ^ ror8(te[(s3 >> 16) & 255]) ^ ror16(te[(s0 >> 8) & 255]) ^
                                ror24(te[s1 & 255]) ^ rk[4 * r + 2];
            const uint32_t t3 = te[s3 >> 24] ^ ror8(te[(s0 >> 16) & 255]) ^ ror16(te[(s1 >> 8) & 255]) ^
                                ror24(te[s2 & 255]) ^ rk[4 * r + 3];
            s0 = t0;
            s1 = t1;
            s2 = t2;
            s3 = t3;
        }
        uint32_t o[4];
        o[0] = ((uint32_t)sb[s0 >> 24] << 24 | (uint32_t)sb[(s1 >> 16) & 255] << 16 | (uint32_t)sb[(s2 >> 8) & 255] << 8 |
                sb[s3 & 255]) ^ rk[40];
        o[1] = ((uint32_t)sb[s1 >> 24] << 24 | (uint32_t)sb[(s2 >> 16) & 255] << 16 | (uint32_t)sb[(s3 >> 8) & 255] << 8 |
                sb[s0 & 255]) ^ rk[41];
        o[2] = ((uint32_t)sb[s2 >> 24] << 24 | (uint32_t)sb[(s3 >> 16) & 255] << 16 | (uint32_t)sb[(s0 >> 8) & 255] << 8 |
                sb[s1 & 255]) ^ rk[42];
        o[3] = ((uint32_t)sb[s3 >> 24] << 24 | (uint32_t)sb[(s0 >> 16) & 255] << 16 | (uint32_t)sb[(s1 >> 8) & 255] << 8 |
                sb[s2 & 255]) ^ rk[43];
        for (int i = 0; i < 16; i++) buf[(blk - nblk_main) * 16 + i] = (uint8_t)(o[i >> 2] >> (24 - 8 * (i & 3)));
    }
    // write only after every tail block is computed (the key may sit in these bytes)
    uint8_t *out = row + out_off + (size_t)nblk_main * 16;
    const uint32_t nb = nbytes - nblk_main * 16;
    for (uint32_t i = 0; i < nb; i++) out[i] = buf[i];
}

}  // namespace mayo
