// mma_perm.cpp -- host check of the tensor-core permutations' tables
// (zeknox_b200/csrc/mma_tables.h): the permutations computed from the tables
// in the order of hash_mma.cuh, every product a sum of byte products as the
// tensor core takes them and the sums recombined in 32-bit words as
// mma_combine does, against the plain permutations of hash.cuh.
// Prints the number of states checked, or the first mismatch (exit code 1).
#include <cstdio>

#include "../../zeknox_b200/csrc/hash.cuh"
#include "../../zeknox_b200/csrc/mma_tables.h"

using namespace zk;

// mma_combine: pairs of sums in 32-bit words, then the sum of the four words
static uint64_t combine(const uint64_t s[8])
{
    unsigned __int128 v = 0;
    for (int i = 0; i < 4; i++) {
        const uint32_t u = (uint32_t)s[2 * i] + (uint32_t)s[2 * i + 1] * 256u;
        v += (unsigned __int128)u << (16 * i);
    }
    return gl_reduce128((uint64_t)v, (uint64_t)(v >> 64));
}

static uint64_t combine_exact(const uint64_t s[8])
{
    unsigned __int128 v = 0;
    for (int i = 0; i < 8; i++) v += (unsigned __int128)s[i] << (8 * i);
    return gl_reduce128((uint64_t)v, (uint64_t)(v >> 64));
}

// the largest sums the recombination takes, and that one more wraps
static bool limit_holds()
{
    const uint64_t top = ((1ULL << 32) - 1) / 257;
    if (!mma_sums_fit(top) || mma_sums_fit(top + 1)) return false;
    uint64_t s[8];
    for (uint64_t &x : s) x = top;
    if (combine(s) != combine_exact(s)) return false;
    for (uint64_t &x : s) x = top + 1;
    return combine(s) != combine_exact(s);
}

// one group of four outputs: `kbs` k-blocks of input lanes, word offsets of
// the operands and the starting sums
static bool group(const MmaTables &t, unsigned tab, unsigned cst, int kbs, const uint64_t *lanes, uint64_t out[4])
{
    for (int o = 0; o < 4; o++) {
        uint64_t sums[8];
        for (int byte = 0; byte < 8; byte++) {
            const int i = byte >> 1, g = 2 * o + (byte & 1);
            uint64_t &s = sums[byte];
            s = t.w[cst + (i * 4 + o) * 4 + (byte & 1)];
            if (s != t.w[cst + (i * 4 + o) * 4 + 2 + (byte & 1)]) return false;
            for (int kb = 0; kb < kbs; kb++)
                for (int q = 0; q < 4; q++)
                    for (int k = 0; k < 8; k++) {
                        const unsigned w = t.w[tab + kb * MMA_KB + ((i >> 1) * 32 + 4 * g + q) * 4 + 2 * (i & 1) + (k >> 2)];
                        s += ((lanes[4 * kb + q] >> (8 * k)) & 255) * ((w >> (8 * (k & 3))) & 255);
                    }
            if (s > t.worst_sum) return false;
        }
        out[o] = combine(sums);
    }
    return true;
}

// one group of a full-round layer: one k-block per pair of byte columns
static bool full_group(const MmaTables &t, unsigned tab, unsigned cst, const uint64_t *lanes, uint64_t out[4])
{
    for (int o = 0; o < 4; o++) {
        uint64_t sums[8];
        for (int byte = 0; byte < 8; byte++) {
            const int i = byte >> 1, g = 2 * o + (byte & 1);
            uint64_t &s = sums[byte];
            s = t.w[cst + (i * 4 + o) * 4 + (byte & 1)];
            for (int q = 0; q < 4; q++) {
                const unsigned *w = &t.w[tab + ((i >> 1) * 32 + 4 * g + q) * 4 + 2 * (i & 1)];
                const unsigned h = 32 * (i >> 1), p = 16 * (i & 1);
                const unsigned a0 = ((unsigned)(lanes[q] >> (h + p)) & 0xFFFF) | ((unsigned)(lanes[4 + q] >> (h + p)) & 0xFFFF) << 16;
                const unsigned a2 = (unsigned)(lanes[8 + q] >> h);
                for (int k = 0; k < 4; k++)
                    s += ((a0 >> (8 * k)) & 255) * ((w[0] >> (8 * k)) & 255) + ((a2 >> (8 * k)) & 255) * ((w[1] >> (8 * k)) & 255);
            }
            if (s > t.worst_sum) return false;
        }
        out[o] = combine(sums);
    }
    return true;
}

static bool permute_tables(const MmaTables &t, int hash, uint64_t s[12])
{
    uint64_t z[36], n[12];
    const uint64_t *rc = hash == 0 ? h_POSEIDON_RC : h_POSEIDON2_RC;
    auto layer = [&](int idx) {
        for (int j = 0; j < 3; j++)
            if (!full_group(t, MMA_FULL + j * MMA_KB, MMA_CONST + (3 * idx + j) * MMA_GROUP, s, n + 4 * j)) return false;
        for (int i = 0; i < 12; i++) s[i] = n[i];
        return true;
    };
    if (hash == 0) for (int i = 0; i < 12; i++) s[i] = gl_add(gl_canon(s[i]), rc[i]);
    else if (!layer(0)) return false;
    for (int f = 0; f < 8; f++) {
        for (int i = 0; i < 12; i++) s[i] = gl_sbox7(gl_canon(s[i]));
        if (f != 3) {
            if (!layer(f + 1)) return false;
            continue;
        }
        for (int i = 0; i < 12; i++) z[i] = s[i];
        for (int b = 0, before = 0; b < 6; before += 3 + b++) {
            uint64_t y[4];
            if (!group(t, MMA_Y + before * MMA_KB, MMA_YCONST + b * MMA_GROUP, 3 + b, z, y)) return false;
            for (int o = 0; o < 4; o++) {
                for (int j = 0; j < o; j++) y[o] = gl_add(y[o], gl_mul(t.h[o - j - 1], z[12 + 4 * b + j]));
                z[12 + 4 * b + o] = 4 * b + o < 22 ? gl_sbox7(y[o]) : ~0ULL;  // no coefficient reads the last two
            }
        }
        for (int j = 0; j < 3; j++)
            if (!group(t, MMA_W + 9 * j * MMA_KB, MMA_CONST + (12 + j) * MMA_GROUP, 9, z, s + 4 * j)) return false;
    }
    return true;
}

// permute_mma_monolith
static bool monolith_tables(const MmaTables &t, uint64_t s[12])
{
    for (int st = 0; st < 7; st++) {
        uint64_t n[12];
        for (int j = 0; j < 3; j++)
            if (!full_group(t, MMA_FULL + j * MMA_KB, MMA_MONO_CONST + (3 * st + j) * MMA_GROUP, s, n + 4 * j)) return false;
        if (st < 6)
            for (int i = 0; i < 4; i++) n[i] = mono_bar(gl_canon(n[i]));
        for (int i = 0; i < 12; i++) s[i] = st < 6 && i ? gl_add(gl_canon(n[i]), gl_mul(n[i - 1], n[i - 1])) : gl_canon(n[i]);
    }
    return true;
}

int main()
{
    if (!limit_holds()) {
        printf("the sums' limit is not the recombination's\n");
        return 1;
    }
    const uint64_t corner[] = {0, 1, 2, GL_P - 1, GL_P - 2, GL_EPS, GL_EPS + 1, 1ULL << 63, GL_P, GL_P + 1, ~0ULL, ~0ULL - 1};
    const int nc = sizeof corner / sizeof *corner;
    uint64_t seed = 12345;
    auto rnd = [&]() {
        seed = seed * 6364136223846793005ULL + 1442695040888963407ULL;
        return seed ^ (seed >> 29);
    };
    int checked = 0;
    for (int hash : {0, 3, 4}) {
        const MmaTables t = hash == 4 ? make_mma_monolith() : make_mma_tables(hash);
        for (int c = 0; c < 3 * nc; c++) {
            uint64_t a[12], b[12];
            for (int i = 0; i < 12; i++)
                a[i] = b[i] = c < nc ? corner[c] : c < 2 * nc ? corner[(c + 5 * i) % nc] : rnd();
            if (hash == 0) poseidon_permute(a);
            else if (hash == 3) poseidon2_permute(a);
            else monolith_permute(a);
            if (!(hash == 4 ? monolith_tables(t, b) : permute_tables(t, hash, b))) {
                printf("hash %d: a byte-column sum above worst_sum, or unequal starting sums\n", hash);
                return 1;
            }
            for (int i = 0; i < 12; i++)
                if (gl_canon(a[i]) != gl_canon(b[i])) {
                    printf("hash %d state %d lane %d differs\n", hash, c, i);
                    return 1;
                }
            checked++;
        }
    }
    printf("%d states\n", checked);
    return 0;
}
