// op_verify.cu -- batched MAYO verify on B200 (reference src/verify.cu:9-212): one CTA or cluster per
// instance, or one CTA per group of instances with long messages, running verify_instance
// (verify_body.cuh).
#include "ops.h"
#include "verify_body.cuh"

namespace mayo {

template <int SET, int CL>
__global__ void __launch_bounds__(VerifyCfg<SET, CL>::NT, VerifyCfg<SET, CL>::MINB) verify_kernel(const VerifyIO io) {
    extern __shared__ __align__(16) uint8_t smem[];
    const size_t inst = blockIdx.x / CL;
    verify_instance<SET, CL>(smem, threadIdx.x, io.epk + inst * io.epk_stride, io.m.ptr(inst), io.m.len(inst),
                             io.sig + inst * io.sig_stride, io.res + inst * io.res_stride,
                             CL > 1 ? (int)cluster_rank() : 0);
}

// Long messages.  One warp hashes a message, 3.1 us per 136 bytes, beside its instance's products; past
// VerifyLong::len bytes that takes longer than they do and the CTA waits, of which an SM holds three
// (MAYO_1) or one.  Then, in a batch of more than one wave, a CTA takes a group of instances: it hashes
// their messages first, one per warp, and does their products one after another.
// us one by one / by groups, at 4,096, 8,192 and 32,768 bytes:
//   MAYO_1   500  274 / 250,   468 / 327,   1,622 / 947;     4,096  1,414 / 1,199, 2,466 / 1,555,  8,776 / 3,713
//   MAYO_3   300  405 / 305,   716 / 420,   2,515 / 1,088;   4,096  3,707 / 2,147, 6,512 / 2,646, 23,288 / 5,673
//   MAYO_5   300      -      761 / 599, 2,565 / 1,205;  4,096      -         7,076 / 4,422, 23,876 / 7,028
// The lines lie where the two meet in batches of two waves, which gain least (MAYO_1, 450: 3,072 bytes 218 /
// 219; MAYO_3, 149: 2,049 160 / 173, 3,072 202 / 197; MAYO_5, 149: 6,145 395 / 421, 8,192 492 / 470).  MAYO_2's six CTAs per SM hash side by
// side as it is.  By the host's length only: with lengths on the device either kernel would have to
// look at each, which cost short messages 0.3 to 12 %.
template <int SET>
struct VerifyLong {
    static constexpr size_t len = SET == 1 ? 3328 : SET == 2 ? ~size_t(0) : SET == 3 ? 3072 : 7168;
};
template <int SET>
static bool verify_is_long(const MsgIO &m) {
    return !m.msg_len && m.mlen > VerifyLong<SET>::len;
}

// Instances group * blockIdx.x .. + group - 1 (group <= CW).
template <int SET>
__global__ void __launch_bounds__(VerifyCfg<SET>::NT, VerifyCfg<SET>::MINB)
    verify_group_kernel(const VerifyIO io, uint32_t batch, uint32_t group) {
    extern __shared__ __align__(16) uint8_t smem[];
    using S = Set<SET>;
    using C = VerifyCfg<SET>;
    static_assert(S::digest / 4 <= 32 && C::CW * S::digest <= C::off_key, "a word per lane; room for the digests");
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t first = blockIdx.x * group, end = min(first + group, batch), own = first + warp;
    uint32_t word = 0;  // of the digest of message `own`
    if (own < end) {
        uint8_t *digest = smem + warp * S::digest;
        WarpKeccak wk;
        wk.setup((int)lane);
        warp_shake<136>(digest, S::digest, io.m.ptr(own), io.m.mlen, wk, (int)lane);
        if (lane < S::digest / 4) word = reinterpret_cast<const uint32_t *>(digest)[lane];
    }
#pragma unroll 1
    for (uint32_t i = first; i < end; i++) {
        __syncthreads();  // the digests are read, the last instance is done
        if (own == i && lane < S::digest / 4) reinterpret_cast<uint32_t *>(smem + C::off_key)[lane] = word;
        verify_instance<SET, 1, true>(smem, threadIdx.x, io.epk + i * io.epk_stride, nullptr, 0,
                                      io.sig + i * io.sig_stride, io.res + i * io.res_stride);
    }
}

template <int SET, int CL>
static int verify_cl(const VerifyIO &io, size_t batch, cudaStream_t st) {
    using C = VerifyCfg<SET, CL>;
    if (!set_smem_attr(verify_kernel<SET, CL>, C::total)) return ST_CUDA;
    return launch_cluster(verify_kernel<SET, CL>, (unsigned)(batch * CL), C::NT, C::total, CL, st, io) == cudaSuccess
               ? ST_OK
               : ST_CUDA;
}

// One CTA per instance or, for long messages, per group: the smallest groups that take no more waves of
// CTAs than groups of CW (2,072 MAYO_1 of 4,096 bytes: three 691 CTAs, 686 us; four 518 CTAs, 771 us).
template <int SET>
static int verify_ctas(const VerifyIO &io, size_t batch, cudaStream_t st) {
    using C = VerifyCfg<SET>;
    if constexpr (SET != 2) {
        if (verify_is_long<SET>(io.m)) {
            int sms = 0;
            if (!device_sms(sms)) return ST_CUDA;
            const size_t slots = (size_t)C::MINB * (size_t)sms, most = (size_t)C::CW * slots;
            const size_t ctas = (batch + most - 1) / most * slots, group = (batch + ctas - 1) / ctas;
            if (group > 1) {
                if (!set_smem_attr(verify_group_kernel<SET>, C::total)) return ST_CUDA;
                verify_group_kernel<SET><<<(unsigned)((batch + group - 1) / group), C::NT, C::total, st>>>(
                    io, (uint32_t)batch, (uint32_t)group);
                return cudaPeekAtLastError() == cudaSuccess ? ST_OK : ST_CUDA;
            }
        }
    }
    return verify_cl<SET, 1>(io, batch, st);
}

template <int SET>
static int verify_t(const VerifyIO &io, size_t batch, cudaStream_t st) {
    // a remainder of long messages has no launch of its own: it would wait for the first one's hashes
    const int per_sm = SET == 2 || verify_is_long<SET>(io.m) ? 0 : VerifyCfg<SET>::MINB;
    return launch_waves(batch, per_sm, ~size_t(0), [&](int cl, size_t first, size_t n) {
        switch (cl) {
            case 8: return verify_cl<SET, 8>(io.from(first), n, st);
            case 4: return verify_cl<SET, 4>(io.from(first), n, st);
            case 2: return verify_cl<SET, 2>(io.from(first), n, st);
            default: return verify_ctas<SET>(io.from(first), n, st);
        }
    });
}

int launch_verify_io(int set, const VerifyIO &io, size_t batch, cudaStream_t st) {
    if (batch == 0) return ST_OK;
    switch (set) {
        case 1: return verify_t<1>(io, batch, st);
        case 2: return verify_t<2>(io, batch, st);
        case 3: return verify_t<3>(io, batch, st);
        case 5: return verify_t<5>(io, batch, st);
        default: return ST_BAD_SET;
    }
}

int launch_verify(int set, uint8_t *pool, size_t pitch, size_t batch, cudaStream_t st, size_t mlen, size_t msg_off,
                  size_t sig_off, size_t res_off) {
    VerifyIO io{pool, pitch, MsgIO{pool + msg_off, pitch, nullptr, nullptr, (uint32_t)mlen}, pool + sig_off, pitch,
                pool + res_off, pitch};
    return launch_verify_io(set, io, batch, st);
}

}  // namespace mayo
