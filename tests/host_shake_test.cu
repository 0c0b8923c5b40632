// Host-side check of the words that a warp's SHAKE sponge absorbs (shake_word in
// cumayo_b200/csrc/common.cuh), at lengths around the rate, 2^31 and 2^32 - 1.  Built and run by
// tests/test_host_shake.py; prints "OK" or the first failing case.
#include <sys/mman.h>

#include <cstdint>
#include <cstdio>

#include "common.cuh"

using namespace mayo;

// The length parameter holds every 32-bit length.
template <class OutLen, class Len>
constexpr bool holds_32_bits(void (*)(uint8_t *, OutLen, const uint8_t *, Len, const WarpKeccak &, int)) {
    return (Len)0xFFFFFFFFu > (Len)0x7FFFFFFFu;
}
static_assert(holds_32_bits(&warp_shake<136>) && holds_32_bits(&warp_shake<168>), "a signed length");

static uint8_t byte_at(uint64_t i) { return (uint8_t)((i * 2654435761u + 12345u) >> 13); }

// The block that starts at byte `at` of `len` input bytes, padded (FIPS 202, SHAKE), byte by byte.
template <int RATE>
static bool block_ok(const uint8_t *in, uint64_t len, uint64_t at) {
    for (int lane = 0; lane < RATE / 8; lane++) {
        uint64_t want = 0;
        for (int b = 0; b < 8; b++) {
            const uint64_t i = at + 8 * lane + b;
            uint8_t v = i < len ? in[i] : 0;
            if (len - at < RATE) {
                if (i == len) v ^= 0x1F;
                if (8 * lane + b == RATE - 1) v ^= 0x80;
            }
            want |= (uint64_t)v << (8 * b);
        }
        if (shake_word<RATE>(in + at, (uint32_t)(len - at), lane) != want) {
            printf("rate %d length %llu block at %llu word %d\n", RATE, (unsigned long long)len, (unsigned long long)at, lane);
            return false;
        }
    }
    return true;
}

// The first blocks, those around 2^31 and the last ones, which hold random bytes.
template <int RATE>
static bool length_ok(uint8_t *in, uint64_t len) {
    const uint64_t last = len / RATE, mid = (1ull << 31) / RATE;
    for (uint64_t b : {(uint64_t)0, (uint64_t)1, mid - 1, mid, mid + 1, last - 1, last}) {
        if (b > last) continue;
        for (uint64_t i = b * RATE; i < (b + 1) * RATE; i++) in[i] = byte_at(i);  // past the input too
        if (!block_ok<RATE>(in, len, b * RATE)) return false;
    }
    return true;
}

int main() {
    const size_t size = (1ull << 32) + 4096;  // mostly untouched pages
    void *m = mmap(nullptr, size, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
    if (m == MAP_FAILED) return printf("mmap\n"), 1;
    uint8_t *base = static_cast<uint8_t *>(m);
    for (uint64_t len : {0ull, 1ull, 7ull, 8ull, 9ull, 135ull, 136ull, 137ull, 167ull, 168ull, 169ull, 272ull, 273ull,
                         (1ull << 31) - 1, 1ull << 31, (1ull << 31) + 1, (1ull << 31) + 200, (1ull << 32) - 2, (1ull << 32) - 1})
        for (int off = 0; off < 9; off += off < 1 ? 1 : 7)  // 0, 1, 8
            if (!length_ok<136>(base + off, len) || !length_ok<168>(base + off, len)) return 1;
    printf("OK\n");
    return 0;
}
