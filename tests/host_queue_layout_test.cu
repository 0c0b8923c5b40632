// Host-side check of the shared-memory layout of the work queue's keypair CTA (QueueCfg in
// cumayo_b200/csrc/queue_cfg.cuh).  Built and run by tests/test_host_queue_layout.py; prints "OK" or
// the first failing case.
#include <cstdio>

#include "queue_cfg.cuh"

using namespace mayo;

template <int SET>
static bool set_ok() {
    using Q = QueueCfg<SET, MAYO_B200_OP_KEYPAIR>;
    using C = typename Q::KC;
    const auto fail = [](const char *what) { return printf("MAYO_%d: %s\n", SET, what), false; };
    // seed_pk is read while P3 starts: beside everything that P3 writes
    if (Q::seedpk < C::total) return fail("seed_pk inside P3's shared memory");
    if (Q::smem < Q::seedpk + 16) return fail("seed_pk past the CTA's shared memory");
    // O is read by P3: beside the AES tables, round keys and runs
    if (Q::aes_end > C::off_o) return fail("O inside the AES tables");
    if (C::off_ctr < C::off_o + Set<SET>::o_bytes) return fail("the work counter inside O");
    // the CTAs per SM that the registers are bounded for (228 KB of shared memory, 1 KB reserved per CTA)
    if (Q::MINB * (Q::smem + 1024) > 228 * 1024) return fail("CTAs per SM");
    return true;
}

int main() {
    if (!set_ok<1>() || !set_ok<2>() || !set_ok<3>() || !set_ok<5>()) return 1;
    printf("OK\n");
    return 0;
}
