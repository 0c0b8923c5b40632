// op_keygen.cu -- batched keypair, expand-sk and expand-pk on B200.
//
// keypair  (reference src/keypair.cu:10-121):  hash kernel (seed_sk, seed_pk || O) -> AES-CTR kernel
//          (P1 || P2 into the row's scratch) -> P3 kernel.
// expandsk (src/expandsk.cu:9-81): hash kernel (O, seed_pk) -> AES-CTR -> L kernel.
//          (Small batches: the AES-CTR kernel hashes too.)
// expandpk (src/expandpk.cu:9-23): AES-CTR only.
#include "aes.cuh"
#include "keygen_body.cuh"
#include "ops.h"

namespace mayo {

// ---------------------------------------------------------------------------------------------
// Hash kernels: one thread per instance, Keccak state in registers; or, for batches up to
// HASH_WARP_MAX, one warp per instance.  The smallest batches have none: the expansion kernel's
// preparing warps hash (AesDerive).
// ---------------------------------------------------------------------------------------------
// keypair: seed_sk = SHAKE128(LE64(rand_index + 2*inst + 1), SK) (src/keypair.cu:35-45) unless
// `seeded`; then seed_pk || O = SHAKE256(seed_sk) (src/keypair.cu:47-50).  seed_pk goes to pk[0:16];
// O is parked in pk[16 : 16 + O_BYTES] until the P3 kernel overwrites that region.
template <int SET>
__global__ void keypair_hash_kernel(uint8_t *pool, size_t pitch, uint32_t batch, uint64_t rand_index, int seeded) {
    using S = Set<SET>;
    const uint32_t inst = blockIdx.x * blockDim.x + threadIdx.x;
    if (inst >= batch) return;
    uint8_t *row = pool + (size_t)inst * pitch;
    uint8_t *sk = row;
    uint8_t *pk = row + align128(S::sk);
    if (!seeded) {
        const uint64_t ctr = rand_index + (uint64_t)(uint32_t)(2u * inst) + 1;
        uint8_t cb[8];
#pragma unroll
        for (int i = 0; i < 8; i++) cb[i] = (uint8_t)(ctr >> (8 * i));
        Sponge<168> sp;
        sp.init();
        sp.absorb(cb, 8);
        sp.finalize();
        sp.squeeze(sk, S::sk);
    }
    Sponge<136> sp2;
    sp2.init();
    sp2.absorb(sk, S::sk);
    sp2.finalize();
    sp2.squeeze(pk, 16);
    sp2.squeeze(pk + 16, S::o_bytes);
}

// expandsk: seed_pk || O = SHAKE256(seed_sk) (src/expandsk.cu:28-35).  O goes to its esk slot;
// seed_pk is parked in the last 16 bytes of the P region, which the AES tail kernel writes last.
template <int SET>
__global__ void expandsk_hash_kernel(uint8_t *pool, size_t pitch, uint32_t batch) {
    using S = Set<SET>;
    const uint32_t inst = blockIdx.x * blockDim.x + threadIdx.x;
    if (inst >= batch) return;
    uint8_t *row = pool + (size_t)inst * pitch;
    Sponge<136> sp;
    sp.init();
    sp.absorb(row, S::sk);
    sp.finalize();
    sp.squeeze(row + S::sk + S::o_bytes + S::p - 16, 16);
    sp.squeeze(row + S::sk, S::o_bytes);
}

// The same with a warp per instance.
constexpr int HASH_WARPS = 4;
template <int SET>
__global__ void __launch_bounds__(32 * HASH_WARPS)
    keypair_hash_warp_kernel(uint8_t *pool, size_t pitch, uint32_t batch, uint64_t rand_index, int seeded) {
    using S = Set<SET>;
    __shared__ uint64_t s_buf[HASH_WARPS][8];  // the counter, the seed
    const int lane = threadIdx.x & 31;
    const uint32_t inst = blockIdx.x * HASH_WARPS + (threadIdx.x >> 5);
    if (inst >= batch) return;
    uint8_t *row = pool + (size_t)inst * pitch, *pk = row + align128(S::sk);
    uint64_t *buf = s_buf[threadIdx.x >> 5];
    const uint8_t *sk = row;
    WarpKeccak wk;
    wk.setup(lane);
    if (!seeded) {
        if (lane == 0) buf[0] = rand_index + (uint64_t)(uint32_t)(2u * inst) + 1;
        __syncwarp();
        uint8_t *seed = reinterpret_cast<uint8_t *>(buf + 1);
        warp_shake<168>(seed, S::sk, reinterpret_cast<const uint8_t *>(buf), 8, wk, lane);
        for (int i = lane; i < S::sk; i += 32) row[i] = seed[i];
        sk = seed;
    }
    warp_shake<136>(pk, 16 + S::o_bytes, sk, S::sk, wk, lane);
}

template <int SET>
__global__ void __launch_bounds__(32 * HASH_WARPS) expandsk_hash_warp_kernel(uint8_t *pool, size_t pitch, uint32_t batch) {
    using S = Set<SET>;
    __shared__ uint64_t s_out[HASH_WARPS][(16 + S::o_bytes + 7) / 8];
    const int lane = threadIdx.x & 31;
    const uint32_t inst = blockIdx.x * HASH_WARPS + (threadIdx.x >> 5);
    if (inst >= batch) return;
    uint8_t *row = pool + (size_t)inst * pitch, *out = reinterpret_cast<uint8_t *>(s_out[threadIdx.x >> 5]);
    WarpKeccak wk;
    wk.setup(lane);
    warp_shake<136>(out, 16 + S::o_bytes, row, S::sk, wk, lane);
    if (lane < 16) row[S::sk + S::o_bytes + S::p - 16 + lane] = out[lane];
    for (int i = lane; i < S::o_bytes; i += 32) row[S::sk + i] = out[16 + i];
}

// ---------------------------------------------------------------------------------------------
// P3 (keypair) and L (expandsk) kernels: one CTA per instance, or a cluster where the batch is small.
// ---------------------------------------------------------------------------------------------
template <int SET, int CL>
__global__ void __launch_bounds__(KeyCfg<SET, CL>::NT, KeyCfg<SET, CL>::MINB) p3_kernel(uint8_t *pool, size_t pitch) {
    using S = Set<SET>;
    using C = KeyCfg<SET, CL>;
    extern __shared__ __align__(16) uint8_t smem[];
    const int tid = threadIdx.x;
    uint8_t *row = pool + (size_t)(blockIdx.x / CL) * pitch;
    uint8_t *pk = row + align128(S::sk);
    const uint8_t *P1 = pk + align128(S::pk);
    // O is parked in pk[16:]: copy it to shared memory before P3 overwrites that region
    for (int i = tid; i < S::o_bytes; i += C::NT) smem[C::off_o + i] = pk[16 + i];
    __syncthreads();
    p3_instance<SET, CL, true>(smem, tid, P1, pk + 16, CL > 1 ? (int)cluster_rank() : 0);
}

template <int SET, int CL>
__global__ void __launch_bounds__(LCfg<SET, CL>::NT, LCfg<SET, CL>::MINB) l_kernel(uint8_t *pool, size_t pitch) {
    using S = Set<SET>;
    using C = LCfg<SET, CL>;
    extern __shared__ __align__(16) uint8_t smem[];
    const int tid = threadIdx.x;
    uint8_t *row = pool + (size_t)(blockIdx.x / CL) * pitch;
    uint8_t *P1 = row + S::sk + S::o_bytes;
    for (int i = tid; i < S::o_bytes; i += C::NT) smem[C::off_o + i] = row[S::sk + i];
    __syncthreads();
    l_instance<SET, CL>(smem, tid, P1, P1 + S::p1, (int)(blockIdx.x % CL));
}

// ---------------------------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------------------------
// Near-equal chunks per instance: the split whose busiest CTA has the least to do, an item counting
// its blocks and AES_ITEM_COST, a split instance whose key lies in the output the tail kernel.  MAYO_1
// (9,031 blocks) at 1,024: 207, 185, 181, 177 us with items of at most 1,536, 3,072, 6,400 and 12,288
// blocks.  Items of up to a whole MAYO_5 key (52,616) against 12,288: verifyWithepk of 1,024 MAYO_3
// 832 -> 809 us, of 592 MAYO_5 996 -> 965; expand-sk of 148 MAYO_5 387 -> 356; keypair of 777 1,292 -> 1,273.
static uint32_t aes_chunks(uint32_t nblk, size_t batch, uint32_t ctas, uint32_t tail, uint32_t *bpc) {
    uint32_t best = 0;
    uint64_t least = ~0ull;
    const uint32_t least_c = (nblk + AES_BLOCKS_PER_ITEM - 1) / AES_BLOCKS_PER_ITEM;
    for (uint32_t c = least_c; c <= (nblk + AES_WORKERS / 2 - 1) / (AES_WORKERS / 2); c++) {
        const uint32_t n = (nblk + c - 1) / c;
        const uint64_t cost =
            ((uint64_t)batch * c + ctas - 1) / ctas * (n + AES_ITEM_COST) + (c > 1 ? tail : 0);
        if (cost < least) {
            least = cost;
            best = c;
        }
    }
    *bpc = (nblk + best - 1) / best;
    return best;
}

struct AesPlan {
    uint32_t ctas, chunks, bpc;
};
// tail: what the tail kernel costs a split instance (0: none is needed).
static bool aes_plan(uint32_t nbytes, size_t batch, uint32_t tail, AesPlan &p) {
    int sms = 0;
    if (!device_sms(sms)) return false;
    p.ctas = (uint32_t)sms;
    p.chunks = aes_chunks((nbytes + 15) / 16, batch, p.ctas, tail, &p.bpc);
    return true;
}
// The kernel derives the keys itself where each CTA gets one item, so that an instance's hash is on
// every CTA's path once and the rest of its sponge runs beside the encryption: keypair of one MAYO_1
// 38.5 -> 31.2 us (of MAYO_2, whose O takes five more blocks of the sponge, 41.7 -> 43.5), of 72 56.7 ->
// 43.3, of 148 80.0 -> 63.6; expand-sk, whose tail launch goes too, 37.8 -> 27.0 and 63.9 -> 45.8.
// With several items per CTA the one preparing warp's Keccak (5 us an item) holds the workers up:
// MAYO_2 at 1,024 334 us -> 394.
static bool aes_derives(const AesPlan &p, size_t batch) { return batch * p.chunks <= p.ctas; }

// nbytes of keystream for every row, keyed from row + key_off or, with DERIVE, from the seeds.
template <bool DERIVE>
static int aes_main(uint8_t *pool, size_t pitch, size_t batch, cudaStream_t st, size_t key_off, size_t out_off,
                    uint32_t nbytes, const AesPlan &p, const AesDerive &dv) {
    if (!set_smem_attr(aes_ctr_kernel<DERIVE>, AES_SMEM)) return ST_CUDA;
    // 32-bit item numbers: at most 2^24 instances per launch
    for (size_t b0 = 0; b0 < batch; b0 += size_t(1) << 24) {
        const uint32_t nb = (uint32_t)(batch - b0 < (size_t(1) << 24) ? batch - b0 : size_t(1) << 24);
        const uint32_t items = nb * p.chunks;
        aes_ctr_kernel<DERIVE><<<items < p.ctas ? items : p.ctas, AES_THREADS, AES_SMEM, st>>>(
            pool + b0 * pitch, pitch, key_off, out_off, nbytes, p.bpc, p.chunks, items, 128u, dv);
    }
    return cudaPeekAtLastError() == cudaSuccess ? ST_OK : ST_CUDA;
}

// nbytes of keystream keyed from row + key_off.  Where the key lies in the output, its blocks may be
// written once nothing is left to read it: by the item itself if it is its instance's only one (its
// workers start after the key schedule), else by the tail kernel.  One launch instead of two: keypair
// of 1,024 MAYO_1 329 -> 317 us, verifyWithepk 371 -> 355, signWithesk's expansion 412 -> 395.
static int aes_expand(uint8_t *pool, size_t pitch, size_t batch, cudaStream_t st, size_t key_off, size_t out_off,
                      uint32_t nbytes, bool key_in_output) {
    AesPlan plan;
    // where there is a tail kernel, the main kernel writes the whole blocks that do not touch the key
    const uint32_t nblk_main = key_in_output ? min(nbytes / 16, (uint32_t)((key_off - out_off) / 16)) : 0;
    const uint32_t tail = key_in_output ? AES_TAIL_COST + AES_TAIL_BLOCK_COST * ((nbytes + 15) / 16 - nblk_main) : 0;
    if (!aes_plan(nbytes, batch, tail, plan)) return ST_CUDA;
    if (!key_in_output || plan.chunks == 1)
        return aes_main<false>(pool, pitch, batch, st, key_off, out_off, nbytes, plan, AesDerive{});
    if (!aes_plan(nblk_main * 16, batch, tail, plan)) return ST_CUDA;
    const int rc = aes_main<false>(pool, pitch, batch, st, key_off, out_off, nblk_main * 16, plan, AesDerive{});
    if (rc != ST_OK) return rc;
    aes_ctr_tail_kernel<<<(unsigned)((batch + AES_TAIL_THREADS - 1) / AES_TAIL_THREADS), AES_TAIL_THREADS, 0, st>>>(
        pool, pitch, key_off, out_off, nblk_main, nbytes, (uint32_t)batch);
    return cudaPeekAtLastError() == cudaSuccess ? ST_OK : ST_CUDA;
}

template <int SET, int CL>
static int p3_cl(uint8_t *pool, size_t pitch, size_t batch, cudaStream_t st) {
    using C = KeyCfg<SET, CL>;
    if (!set_smem_attr(p3_kernel<SET, CL>, C::total)) return ST_CUDA;
    return launch_cluster(p3_kernel<SET, CL>, (unsigned)(batch * CL), C::NT, C::total, CL, st, pool, pitch) == cudaSuccess
               ? ST_OK
               : ST_CUDA;
}
// The CTAs of an instance share no shared memory here: a plain grid.
template <int SET, int CL>
static int l_cl(uint8_t *pool, size_t pitch, size_t batch, cudaStream_t st) {
    using C = LCfg<SET, CL>;
    if (!set_smem_attr(l_kernel<SET, CL>, C::total)) return ST_CUDA;
    l_kernel<SET, CL><<<(unsigned)(batch * CL), C::NT, C::total, st>>>(pool, pitch);
    return cudaPeekAtLastError() == cudaSuccess ? ST_OK : ST_CUDA;
}

template <int SET>
static int keypair_t(uint8_t *pool, size_t pitch, size_t batch, cudaStream_t st, uint64_t rand_index, bool seeded) {
    using S = Set<SET>;
    const size_t pk_off = align128(S::sk), p_off = pk_off + align128(S::pk);
    int rc;
    AesPlan plan;
    if (!aes_plan(S::p, batch, 0, plan)) return ST_CUDA;
    if (aes_derives(plan, batch)) {
        rc = aes_main<true>(pool, pitch, batch, st, pk_off, p_off, S::p, plan,
                      AesDerive{(uint32_t)S::sk, (uint32_t)S::o_bytes, 1u, seeded ? 0u : 1u, pk_off + 16, rand_index});
    } else {
        if (batch <= HASH_WARP_MAX)
            keypair_hash_warp_kernel<SET><<<(unsigned)((batch + HASH_WARPS - 1) / HASH_WARPS), 32 * HASH_WARPS, 0, st>>>(
                pool, pitch, (uint32_t)batch, rand_index, seeded ? 1 : 0);
        else
            keypair_hash_kernel<SET><<<(unsigned)((batch + 127) / 128), 128, 0, st>>>(pool, pitch, (uint32_t)batch,
                                                                                         rand_index, seeded ? 1 : 0);
        rc = aes_expand(pool, pitch, batch, st, pk_off, p_off, S::p, false);
    }
    if (rc) return rc;
    return launch_waves(batch, SET == 2 ? 0 : KeyCfg<SET>::MINB, ~size_t(0), [&](int cl, size_t first, size_t n) {
        switch (cl) {
            case 8: return p3_cl<SET, 8>(pool + first * pitch, pitch, n, st);
            case 4: return p3_cl<SET, 4>(pool + first * pitch, pitch, n, st);
            case 2: return p3_cl<SET, 2>(pool + first * pitch, pitch, n, st);
            default: return p3_cl<SET, 1>(pool + first * pitch, pitch, n, st);
        }
    });
}

template <int SET>
static int expandsk_t(uint8_t *pool, size_t pitch, size_t batch, cudaStream_t st) {
    using S = Set<SET>;
    const size_t out_off = S::sk + S::o_bytes;
    int rc;
    AesPlan plan;
    if (!aes_plan(S::p, batch, 0, plan)) return ST_CUDA;
    if (aes_derives(plan, batch)) {
        rc = aes_main<true>(pool, pitch, batch, st, 0, out_off, S::p, plan,
                      AesDerive{(uint32_t)S::sk, (uint32_t)S::o_bytes, 0u, 0u, (size_t)S::sk, 0});
    } else {
        if (batch <= HASH_WARP_MAX)
            expandsk_hash_warp_kernel<SET><<<(unsigned)((batch + HASH_WARPS - 1) / HASH_WARPS), 32 * HASH_WARPS, 0, st>>>(
                pool, pitch, (uint32_t)batch);
        else
            expandsk_hash_kernel<SET><<<(unsigned)((batch + 127) / 128), 128, 0, st>>>(pool, pitch, (uint32_t)batch);
        rc = aes_expand(pool, pitch, batch, st, out_off + S::p - 16, out_off, S::p, true);
    }
    if (rc) return rc;
    return launch_waves(batch, LCfg<SET>::MINB, ~size_t(0), [&](int cl, size_t first, size_t n) {
        switch (cl) {
            case 8: return l_cl<SET, 8>(pool + first * pitch, pitch, n, st);
            case 4: return l_cl<SET, 4>(pool + first * pitch, pitch, n, st);
            case 2: return l_cl<SET, 2>(pool + first * pitch, pitch, n, st);
            default: return l_cl<SET, 1>(pool + first * pitch, pitch, n, st);
        }
    });
}

template <int SET>
static int expandpk_t(uint8_t *pool, size_t pitch, size_t batch, cudaStream_t st) {
    using S = Set<SET>;
    return aes_expand(pool, pitch, batch, st, S::p - 16, 0, S::p, true);
}

#define MAYO_DISPATCH(set, call)             \
    switch (set) {                           \
        case 1: { constexpr int SET = 1; return call; } \
        case 2: { constexpr int SET = 2; return call; } \
        case 3: { constexpr int SET = 3; return call; } \
        case 5: { constexpr int SET = 5; return call; } \
        default: return ST_BAD_SET;          \
    }

int launch_keypair(int set, uint8_t *pool, size_t pitch, size_t batch, cudaStream_t st, uint64_t rand_index) {
    if (batch == 0) return ST_OK;
    MAYO_DISPATCH(set, (keypair_t<SET>(pool, pitch, batch, st, rand_index, false)))
}
int launch_keypair_seeded(int set, uint8_t *pool, size_t pitch, size_t batch, cudaStream_t st) {
    if (batch == 0) return ST_OK;
    MAYO_DISPATCH(set, (keypair_t<SET>(pool, pitch, batch, st, 0, true)))
}
int launch_expandsk(int set, uint8_t *pool, size_t pitch, size_t batch, cudaStream_t st) {
    if (batch == 0) return ST_OK;
    MAYO_DISPATCH(set, (expandsk_t<SET>(pool, pitch, batch, st)))
}
int launch_expandpk(int set, uint8_t *pool, size_t pitch, size_t batch, cudaStream_t st) {
    if (batch == 0) return ST_OK;
    MAYO_DISPATCH(set, (expandpk_t<SET>(pool, pitch, batch, st)))
}

}  // namespace mayo
