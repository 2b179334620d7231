// gen_mma_tables.cpp -- build step: writes the tables of mma_tables.h, and
// Poseidon-BN128's constants in 29-bit limbs (bn254_29.cuh), as C initialiser
// lists to standard output.
#include <stdio.h>

#include "bn254.cuh"
#include "mma_tables.h"

static void print_tables(const char *name, const zk::MmaTables &t)
{
    for (int d = 0; d < 3; d++) printf("#define ZK_MMA_%s_H%d 0x%016llxULL\n", name, d + 1, (unsigned long long)t.h[d]);
    printf("#define ZK_MMA_%s_LIST \\\n", name);
    for (size_t i = 0; i < t.w.size(); i++)
        printf("0x%x,%s", t.w[i], i + 1 == t.w.size() ? "\n" : i % 16 == 15 ? " \\\n" : "");
}

// x 2^256 mod r -> x 2^261 mod r in nine limbs of 29 bits, appended
static void push29(std::vector<uint32_t> &out, zk::Fr x, int doublings)
{
    for (int d = 0; d < doublings; d++) x = zk::fr_add(x, x);
    for (int k = 0; k < 9; k++) {
        const int bit = 29 * k, q = bit >> 5, sh = bit & 31;
        uint64_t v = x.w[q];
        if (q + 1 < 8) v |= (uint64_t)x.w[q + 1] << 32;
        out.push_back((uint32_t)(v >> sh) & ((1u << 29) - 1));
    }
}

static void print_fr29()
{
    static const uint32_t c[800] = {ZK_BN128_C_LIST}, s[4320] = {ZK_BN128_S_LIST}, m[200] = {ZK_BN128_M_LIST}, p[200] = {ZK_BN128_P_LIST};
    std::vector<uint32_t> t, r;
    zk::Fr x;
    auto table = [&](const uint32_t *w, int elements) {
        for (int e = 0; e < elements; e++) {
            for (int k = 0; k < 8; k++) x.w[k] = w[8 * e + k];
            push29(t, x, 5);
        }
    };
    table(c, 100);
    table(s, 540);
    table(m, 25);
    table(p, 25);
    for (int k = 0; k < 8; k++) x.w[k] = zk::bn_r2_limb(k);
    push29(t, x, 10);  // 2^512 -> 2^522
    for (int k = 0; k < 8; k++) x.w[k] = zk::bn_r_limb(k);
    push29(r, x, 0);
    printf("#define ZK_FR29_NP 0x%xu\n#define ZK_FR29_WORDS %zu\n#define ZK_FR29_R_LIST ", ZK_BN254_NP & ((1u << 29) - 1), t.size());
    for (size_t i = 0; i < r.size(); i++) printf("0x%xu%s", r[i], i + 1 < r.size() ? ", " : "\n");
    printf("#define ZK_FR29_LIST \\\n");
    for (size_t i = 0; i < t.size(); i++) printf("0x%x,%s", t[i], i + 1 == t.size() ? "\n" : i % 16 == 15 ? " \\\n" : "");
}

int main()
{
    printf("// written by gen_mma_tables.cpp\n#pragma once\n");
    static const uint64_t rc[360] = {ZK_POSEIDON_RC_LIST};
    printf("#define ZK_MMA_POSEIDON_RC0");
    for (int i = 0; i < 12; i++) printf(" 0x%016llxULL%s", (unsigned long long)rc[i], i < 11 ? "," : "\n");
    print_tables("POSEIDON", zk::make_mma_tables(0));
    print_tables("POSEIDON2", zk::make_mma_tables(3));
    print_tables("MONOLITH", zk::make_mma_monolith());
    print_fr29();
    return 0;
}
