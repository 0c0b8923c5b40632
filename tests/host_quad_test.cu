// Host-side checks of the products on quads of key rows (cumayo_b200/csrc/quad.cuh), whose pieces are
// __host__ __device__.  Built and run by tests/test_host_quad.py; prints "OK" or the first failing case.
#include <cstdint>
#include <cstdio>

#include "quad.cuh"

using namespace mayo;

static uint32_t ref_mul(uint32_t a, uint32_t b) {  // carry-less product mod x^4 + x + 1
    uint32_t r = 0;
    for (int i = 0; i < 4; i++)
        if (b >> i & 1) r ^= a << i;
    for (int d = 6; d >= 4; d--)
        if (r >> d & 1) r ^= 0x13u << (d - 4);
    return r & 0xF;
}
static uint64_t state = 88172645463325252ull;
static uint32_t rnd() {
    state ^= state << 13;
    state ^= state >> 7;
    state ^= state << 17;
    return (uint32_t)state;
}
static uint32_t nib(uint32_t w, int c) { return w >> (4 * c) & 0xF; }
// coordinate e of row i of a quad's planes: bit 4 e + i of each
static uint32_t entry(const G4 &v, int e, int i) {
    const int b = 4 * e + i;
    return (v.p0 >> b & 1) | (v.p1 >> b & 1) << 1 | (v.p2 >> b & 1) << 2 | (v.p3 >> b & 1) << 3;
}
#define FAIL(...)            \
    do {                     \
        printf(__VA_ARGS__); \
        printf("\n");        \
        return 1;            \
    } while (0)

int main() {
    // the nine forms of a product: every pair of scalars, in every bit position
    for (uint32_t a = 0; a < 16; a++)
        for (uint32_t b = 0; b < 16; b++) {
            const uint4 ma = scalar_masks(a), mb = scalar_masks(b);
            uint32_t fa[NFORM], fb[NFORM], A[NFORM];
            forms_of(G4{ma.x, ma.y, ma.z, ma.w}, fa);
            forms_of(G4{mb.x, mb.y, mb.z, mb.w}, fb);
            for (int d = 0; d < NFORM; d++) A[d] = fa[d] & fb[d];
            const G4 p = forms_fold(A);
            const uint4 want = scalar_masks(ref_mul(a, b));
            if (p.p0 != want.x || p.p1 != want.y || p.p2 != want.z || p.p3 != want.w) FAIL("product %u %u", a, b);
        }
    for (int it = 0; it < 2000; it++) {
        const uint32_t w[4] = {rnd(), rnd(), rnd(), rnd()};
        const G4 v = quad_planes(w[0], w[1], w[2], w[3]);
        for (int e = 0; e < 8; e++)
            for (int i = 0; i < 4; i++)
                if (entry(v, e, i) != nib(w[i], e)) FAIL("quad_planes it=%d e=%d i=%d", it, e, i);
        const G4 back = quad_planes(v.p0, v.p1, v.p2, v.p3);
        if (back.p0 != w[0] || back.p1 != w[1] || back.p2 != w[2] || back.p3 != w[3]) FAIL("quad_planes is its own inverse");
        const uint32_t sum = quad_row_sum(v);
        for (int e = 0; e < 8; e++)
            if (nib(sum, e) != (nib(w[0], e) ^ nib(w[1], e) ^ nib(w[2], e) ^ nib(w[3], e))) FAIL("quad_row_sum it=%d e=%d", it, e);
        // a sum of products, its ANDs accumulated and recombined once
        uint32_t A[NFORM] = {}, want[4][8] = {};
        for (int q = 0; q < 7; q++) {
            const uint32_t x[4] = {rnd(), rnd(), rnd(), rnd()}, s = rnd() & 0xF;
            const uint4 m = scalar_masks(s);
            uint32_t f[NFORM], mf[NFORM];
            forms_of(quad_planes(x[0], x[1], x[2], x[3]), f);
            forms_of(G4{m.x, m.y, m.z, m.w}, mf);
            for (int d = 0; d < NFORM; d++) A[d] = lop_xand(A[d], mf[d], f[d]);
            for (int i = 0; i < 4; i++)
                for (int e = 0; e < 8; e++) want[i][e] ^= ref_mul(nib(x[i], e), s);
        }
        const G4 p = forms_fold(A);
        for (int i = 0; i < 4; i++)
            for (int e = 0; e < 8; e++)
                if (entry(p, e, i) != want[i][e]) FAIL("sum of products it=%d e=%d i=%d", it, e, i);
    }
    printf("OK\n");
    return 0;
}
