// op_verify.cu -- batched MAYO verify on B200 (reference src/verify.cu:9-212): one CTA per
// instance running verify_instance (verify_body.cuh).
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

template <int SET, int CL>
static int verify_cl(const VerifyIO &io, size_t batch, cudaStream_t st) {
    using C = VerifyCfg<SET, CL>;
    if (!set_smem_attr(verify_kernel<SET, CL>, C::total)) return ST_CUDA;
    return launch_cluster(verify_kernel<SET, CL>, (unsigned)(batch * CL), C::NT, C::total, CL, st, io) == cudaSuccess
               ? ST_OK
               : ST_CUDA;
}

template <int SET>
static int verify_t(const VerifyIO &io, size_t batch, cudaStream_t st) {
    return launch_waves(batch, SET == 2 ? 0 : VerifyCfg<SET>::MINB, ~size_t(0), [&](int cl, size_t first, size_t n) {
        switch (cl) {
            case 8: return verify_cl<SET, 8>(io.from(first), n, st);
            case 4: return verify_cl<SET, 4>(io.from(first), n, st);
            case 2: return verify_cl<SET, 2>(io.from(first), n, st);
            default: return verify_cl<SET, 1>(io.from(first), n, st);
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
