// queue_cfg.cuh -- the CTA of each (set, op) kernel of the work queue: threads, CTAs per SM, shared
// memory and global scratch.
#pragma once

#include "../../include/mayo_b200.h"
#include "keygen_body.cuh"
#include "sign_body.cuh"
#include "verify_body.cuh"

namespace mayo {

template <int SET, int OP>
struct QueueCfg;

template <int SET>
struct QueueCfg<SET, MAYO_B200_OP_KEYPAIR> {
    using S = Set<SET>;
    // MAYO_2: four warps instead of the batched kernel's two, for the expansion's sake
    using KC = KeyCfg<SET, 1, SET == 2 ? 4 : 0>;
    static constexpr int NT = KC::NT, MINB = KC::MINB;
    // as many replicated round tables as the P3 area below O holds (MAYO_1: T0; MAYO_2: T0 and
    // ror16(T0); MAYO_3: three; MAYO_5: all four) and the round keys; dead once the keystream is written
    static constexpr size_t runs = ((size_t)S::p / 16 + 256) / 256 + 1;  // AesRuns of an instance
    static constexpr size_t aes_bytes(int n) { return (size_t)n * 256 * 32 * 4 + 44 * 4 + 16 * runs; }
    static constexpr int NTAB = KC::off_o >= aes_bytes(4) ? 4 : KC::off_o >= aes_bytes(3) ? 3 : KC::off_o >= aes_bytes(2) ? 2 : 1;
    static constexpr size_t run = (size_t)NTAB * 256 * 32 * 4 + 44 * 4;  // after the round keys (16-byte aligned)
    static constexpr size_t aes_end = aes_bytes(NTAB);
    static_assert(KC::off_o >= aes_end, "O must not overlap the AES tables");
    // seed_pk, copied to the public key while P3 starts (and sets its work counter)
    static constexpr size_t seedpk = KC::total;
    static_assert(seedpk >= KC::off_ctr + 16, "seed_pk must not overlap P3's memory");
    static constexpr size_t smem = seedpk + 16;
    static constexpr size_t scratch = pad16((size_t)S::p + 16);  // P1 || P2 of one keypair
};

template <int SET>
struct QueueCfg<SET, MAYO_B200_OP_SIGN> {
    static constexpr int NT = SignCfg<SET>::NT, MINB = SignCfg<SET>::MINB;
    static constexpr size_t smem = SignCfg<SET>::total;
    static constexpr size_t scratch = 0;
};

template <int SET>
struct QueueCfg<SET, MAYO_B200_OP_VERIFY> {
    static constexpr int NT = VerifyCfg<SET>::NT, MINB = VerifyCfg<SET>::MINB;
    static constexpr size_t smem = VerifyCfg<SET>::total;
    static constexpr size_t scratch = 0;
};

}  // namespace mayo
