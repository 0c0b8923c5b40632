// launch_util.cuh -- host-side helpers shared by the launchers.
#pragma once

#include <cuda_runtime.h>
#include <cstddef>

#include "ops.h"

namespace mayo {

__host__ __device__ constexpr size_t pad16(size_t x) { return (x + 15) / 16 * 16; }

// CTAs per instance of the per-instance sign and verify: a batch that leaves SMs idle gives each
// instance a cluster of them, as many as one wave holds (16, 36 and 72 clusters of 8, 4 and 2 run at
// once; 12 and 32 leave room for other work).  MAYO_5 verify, us: batch 8 31 (8 CTAs) against 41
// (4), 18 58 against 41; 24 42 (4) against 63 (2), 36 79 against 64; 72 64 (2) against 109 (1),
// 100 125 against 109.
inline int cluster_ctas(size_t batch) { return batch <= 12 ? 8 : batch <= 32 ? 4 : batch <= 72 ? 2 : 1; }

// Opt `kernel` into `bytes` of dynamic shared memory on the current device.  The attribute is
// per kernel and per device; setting it is a cheap host call that is not a stream operation.
template <class K>
inline bool set_smem_attr(K kernel, size_t bytes) {
    if (bytes <= 48 * 1024) return true;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) == cudaSuccess;
}

// The current device's SMs.
inline bool device_sms(int &sms) {
    int dev = 0;
    return cudaGetDevice(&dev) == cudaSuccess &&
           cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess;
}

// Calls f(cl, first, count) -> status for the launches of a batch.  It is one launch, but up to
// `waves` full waves of one-CTA instances (per_sm CTAs on each SM; 0: never) and a remainder that
// clusters take are two: alone the remainder holds a few SMs for a whole wave's time.  MAYO_5, us:
// verify 149 214 -> 150, 301 328 -> 263, 2,077 1,620 -> 1,574; keypair 149 380 -> 325; expand-sk 149
// 576 -> 442; sign 301 572 -> 525.  Not where an SM's many small CTAs take the remainder up as they
// finish (MAYO_2: verify 900 76.1 -> 76.5, keypair 940 319 -> 327, sign 900 138 -> 153; MAYO_1's three
// in sign: 450 204 -> 254), nor for a signature after more waves than two: the remainder waits for
// every second attempt of the first launch (MAYO_5, 777, five waves: 1,105 -> 1,254; one and two waves
// gained in sign, three and four were not measured).
template <class F>
inline int launch_waves(size_t batch, int per_sm, size_t waves, F f) {
    if (per_sm == 0) return f(cluster_ctas(batch), size_t(0), batch);
    int sms = 0;
    if (!device_sms(sms)) return ST_CUDA;
    const size_t slots = (size_t)per_sm * (size_t)sms, rest = batch % slots;
    if (batch < slots || batch / slots > waves || rest == 0 || cluster_ctas(rest) == 1)
        return f(cluster_ctas(batch), size_t(0), batch);
    const int rc = f(1, size_t(0), batch - rest);
    return rc ? rc : f(cluster_ctas(rest), batch - rest, rest);
}

// Launch `kernel` on clusters of `cl` CTAs (cl = 1: a plain launch); ctas is a multiple of cl.
template <class... P, class... A>
inline cudaError_t launch_cluster(void (*kernel)(P...), unsigned ctas, unsigned threads, size_t smem, unsigned cl,
                                  cudaStream_t st, const A &...args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    if (cl > 1) {
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = cl;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
    }
    return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

}  // namespace mayo
