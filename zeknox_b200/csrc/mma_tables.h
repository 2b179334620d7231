// mma_tables.h -- tables of the tensor-core permutations (hash_mma.cuh),
// computed on the host from the round constants and the linear layers.
//
// A linear layer over Goldilocks is an integer matrix product on bytes: with
// the input lanes split into bytes, x = sum_i 2^(8i) x_i, an output is
//     sum_lanes c x  =  sum_b 2^(8b) sum_(lane, i) x_i * byte_b(c * 2^(8i) mod p),
// so eight byte columns per output lane hold the reduction of every shifted
// coefficient already, and an 8-bit tensor-core product with 32-bit sums gives
// the eight sums exactly.  The largest sums any input can reach are 9,092,025
// (Poseidon), 9,174,390 (Poseidon2) and 41,055 (Monolith), below the
// 16,711,935 that mma_combine's 32-bit words hold (mma_sums_fit).
//
// The 22 partial rounds of Poseidon and Poseidon2 are affine but for the S-box
// on lane 0, so lane 0 before the S-box of partial round r is an affine form
// of the 12 lanes z entering the segment and of the S-box outputs x_0..x_(r-1)
// (the idea of the sparse factorisation of the Poseidon paper, eprint 2019/458
// appendix B, taken to whole rounds).  They run in blocks of four: the forms
// over z and the x of earlier blocks are tensor-core products (Y), the terms
// inside a block multiply-adds with the three coefficients h1..h3 (the same in
// every round: the partial rounds share one matrix), and the lanes entering
// the next full round a last product over z and all x (W).
//
// Operand order (mma.m16n8k32, row x col): thread t = lane & 3 of a quad holds
// bytes 4t..4t+3 and 16+4t..16+4t+3 of a 32-byte k-block, which are here the
// low and high halves of lane 4 kb + t, so a state's registers are the A
// operand as they stand.  Column n of byte pair i of output group j belongs
// to output lane 4j + (n >> 1), byte 2i + (n & 1): thread t then receives all
// eight sums of lane 4j + t.
#pragma once
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>

#include <vector>

#include "gl64.cuh"
#include "mma_layout.h"
#include "zk_constants.h"

namespace zk {

struct MmaTables {
    std::vector<uint32_t> w;  // the words of mma_layout.h
    uint64_t h[3] = {};       // coefficients inside a block of partial rounds
    uint64_t worst_sum = 0;   // largest byte-column sum any input can reach
};

// mma_combine adds 256 times one sum to another in a 32-bit word.
constexpr bool mma_sums_fit(uint64_t worst_sum) { return 257 * worst_sum < (1ULL << 32); }

namespace mma_gen {

struct Form {
    uint64_t z[12] = {}, x[22] = {}, c = 0;
};

inline void axpy(Form &d, uint64_t k, const Form &s)
{
    for (int i = 0; i < 12; i++) d.z[i] = gl_add(d.z[i], gl_mul(k, s.z[i]));
    for (int i = 0; i < 22; i++) d.x[i] = gl_add(d.x[i], gl_mul(k, s.x[i]));
    d.c = gl_add(d.c, gl_mul(k, s.c));
}

// Full-round matrix m[out][in] of hash type h (0 Poseidon, 3 Poseidon2, 4 Monolith).
inline void full_matrix(int h, uint64_t m[12][12])
{
    static const uint32_t pc[12] = {ZK_POSEIDON_CIRC_LIST}, mc[12] = {ZK_MONOLITH_CIRC_LIST};
    static const uint32_t m4[4][4] = {{5, 7, 1, 3}, {4, 6, 1, 1}, {1, 3, 5, 7}, {1, 1, 4, 6}};
    for (int r = 0; r < 12; r++)
        for (int c = 0; c < 12; c++) {
            if (h == 0) m[r][c] = pc[(c - r + 12) % 12] + (r == 0 && c == 0 ? ZK_POSEIDON_DIAG0 : 0);
            else if (h == 4) m[r][c] = mc[(c - r + 12) % 12];
            else m[r][c] = m4[r % 4][c % 4] * (r / 4 == c / 4 ? 2 : 1);
        }
}

// Appends the B operands of one group of four outputs over `kbs` k-blocks;
// coef(o, lane) is the coefficient of input lane `lane` in output o < 4.
template <class F>
void emit_group(MmaTables &t, int kbs, F coef)
{
    uint64_t sums[4][8] = {};
    for (int kb = 0; kb < kbs; kb++)
        for (int np = 0; np < 2; np++)
            for (int lane = 0; lane < 32; lane++) {
                const int g = lane >> 2, q = lane & 3, o = g >> 1;
                for (int half = 0; half < 2; half++) {
                    const int byte = 2 * (2 * np + half) + (g & 1);
                    uint32_t b[2] = {0, 0};
                    uint64_t c = coef(o, 4 * kb + q);
                    for (int i = 0; i < 8; i++) {
                        const uint32_t v = (uint32_t)(c >> (8 * byte)) & 255u;
                        b[i >> 2] |= v << (8 * (i & 3));
                        sums[o][byte] += 255ULL * v;
                        c = gl_mul(c, 256);
                    }
                    t.w.push_back(b[0]);
                    t.w.push_back(b[1]);
                }
            }
    for (auto &r : sums)
        for (uint64_t s : r)
            if (s + 255 > t.worst_sum) t.worst_sum = s + 255;
}

// Appends the B operands of one group of four outputs of a layer whose
// coefficients are below 256: column pair i multiplies bytes 2i, 2i + 1 of
// lanes t and 4 + t (k-bytes 0..3 of thread t) and the word of lane 8 + t they
// are in (k-bytes 16..19).
template <class F>
void emit_full(MmaTables &t, F coef)
{
    uint64_t sums[4][8] = {};
    for (int np = 0; np < 2; np++)
        for (int lane = 0; lane < 32; lane++) {
            const int g = lane >> 2, q = lane & 3, o = g >> 1, odd = g & 1;
            for (int half = 0; half < 2; half++) {
                const int i = 2 * np + half;
                const uint32_t c0 = (uint32_t)coef(o, q), c1 = (uint32_t)coef(o, 4 + q), c2 = (uint32_t)coef(o, 8 + q);
                if ((c0 | c1 | c2) > 255) abort();
                t.w.push_back(c0 << (8 * odd) | c1 << (16 + 8 * odd));
                t.w.push_back(c2 << (16 * (i & 1) + 8 * odd));
                sums[o][2 * i + odd] += 255ULL * (c0 + c1 + c2);
            }
        }
    for (auto &r : sums)
        for (uint64_t s : r)
            if (s + 255 > t.worst_sum) t.worst_sum = s + 255;
}

// Appends the starting sums (the bytes of a constant per output) of one group.
template <class F>
void emit_const(MmaTables &t, F value)
{
    for (int i = 0; i < 4; i++)
        for (int q = 0; q < 4; q++) {
            const uint64_t v = value(q);
            for (int dup = 0; dup < 2; dup++) {
                t.w.push_back((uint32_t)(v >> (16 * i)) & 255u);
                t.w.push_back((uint32_t)(v >> (16 * i + 8)) & 255u);
            }
        }
}

inline void check_sums(const MmaTables &t)
{
    if (!mma_sums_fit(t.worst_sum)) {
        fprintf(stderr, "mma_tables: a byte-column sum can reach %llu\n", (unsigned long long)t.worst_sum);
        abort();
    }
}

inline void expect(const MmaTables &t, size_t words, const char *what)
{
    if (t.w.size() != words) {
        fprintf(stderr, "mma_tables: %s at word %zu, expected %zu\n", what, t.w.size(), words);
        abort();
    }
}

}  // namespace mma_gen

// Tables of Monolith.
inline MmaTables make_mma_monolith()
{
    using namespace mma_gen;
    static const uint64_t rc[84] = {ZK_MONOLITH_RC_LIST};
    uint64_t m[12][12];
    full_matrix(4, m);
    MmaTables t;
    for (int j = 0; j < 3; j++) emit_full(t, [&](int o, int l) { return m[4 * j + o][l]; });
    expect(t, MMA_MONO_CONST, "Monolith constants");
    for (int r = 0; r < 7; r++)
        for (int j = 0; j < 3; j++) emit_const(t, [&](int q) { return rc[12 * r + 4 * j + q]; });
    expect(t, MMA_MONO_WORDS, "end");
    check_sums(t);
    return t;
}

// Tables of Poseidon (0) or Poseidon2 (3).
inline MmaTables make_mma_tables(int hash)
{
    using namespace mma_gen;
    static const uint64_t prc[360] = {ZK_POSEIDON_RC_LIST}, p2rc[360] = {ZK_POSEIDON2_RC_LIST};
    static const uint64_t diag[12] = {ZK_POSEIDON2_DIAG_LIST};
    const uint64_t *rc = hash == 0 ? prc : p2rc;
    uint64_t m[12][12];
    full_matrix(hash, m);
    // the segment: the linear layer of round 3, 22 partial rounds, constants of round 26
    Form lane[12], y[22];
    auto apply_full = [&]() {
        Form n[12];
        for (int r = 0; r < 12; r++)
            for (int c = 0; c < 12; c++) axpy(n[r], m[r][c], lane[c]);
        for (int r = 0; r < 12; r++) lane[r] = n[r];
    };
    for (int i = 0; i < 12; i++) lane[i].z[i] = 1;
    apply_full();
    for (int r = 0; r < 22; r++) {
        for (int i = 0; i < (hash == 0 ? 12 : 1); i++) lane[i].c = gl_add(lane[i].c, rc[12 * (4 + r) + i]);
        y[r] = lane[0];
        lane[0] = Form();
        lane[0].x[r] = 1;
        if (hash == 0) {
            apply_full();
        } else {
            Form sum;
            for (int i = 0; i < 12; i++) axpy(sum, 1, lane[i]);
            for (int i = 0; i < 12; i++) {
                Form n = sum;
                axpy(n, diag[i], lane[i]);
                lane[i] = n;
            }
        }
    }
    for (int i = 0; i < 12; i++) lane[i].c = gl_add(lane[i].c, rc[12 * 26 + i]);

    MmaTables t;
    for (int d = 1; d <= 3; d++) t.h[d - 1] = y[d].x[0];
    for (int r = 0; r < 22; r++)
        for (int j = 4 * (r / 4); j < r; j++)
            if (y[r].x[j] != t.h[r - j - 1]) {
                fprintf(stderr, "mma_tables: partial rounds do not share one matrix\n");
                abort();
            }
    // coefficient of input lane l (z, then x); the two x of the last block that no round makes have none
    auto in = [](const Form &f, int l) -> uint64_t { return l < 12 ? f.z[l] : l < 34 ? f.x[l - 12] : 0; };
    expect(t, MMA_FULL, "full-round matrix");
    for (int j = 0; j < 3; j++) emit_full(t, [&](int o, int l) { return m[4 * j + o][l]; });
    expect(t, MMA_Y, "partial rounds");
    for (int b = 0; b < 6; b++)
        emit_group(t, 3 + b, [&](int o, int l) { return 4 * b + o < 22 ? in(y[4 * b + o], l) : 0; });
    expect(t, MMA_W, "segment output");
    for (int j = 0; j < 3; j++) emit_group(t, 9, [&](int o, int l) { return in(lane[4 * j + o], l); });
    expect(t, MMA_CONST, "layer constants");
    for (int layer = 0; layer < 9; layer++)
        for (int j = 0; j < 3; j++)
            emit_const(t, [&](int q) -> uint64_t {
                const int i = 4 * j + q;
                if (layer < 4) return rc[12 * layer + i];           // before full round `layer`
                if (layer == 4) return lane[i].c;                   // before round 26
                return layer < 8 ? rc[12 * (22 + layer) + i] : 0;   // before rounds 27..29; none after the last
            });
    expect(t, MMA_YCONST, "partial-round constants");
    for (int b = 0; b < 6; b++)
        emit_const(t, [&](int q) -> uint64_t { return 4 * b + q < 22 ? y[4 * b + q].c : 0; });
    expect(t, MMA_WORDS, "end");
    check_sums(t);
    return t;
}

}  // namespace zk
