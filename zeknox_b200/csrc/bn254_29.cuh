// bn254_29.cuh -- F_r (BN254 scalar field) in nine limbs of 29 bits, and
// Poseidon-BN128 on them: the device form of the Merkle kernels.
//
// bn254.cuh multiplies on eight 32-bit limbs, where every row of products is a
// carry chain: a forest of 2^14 leaves, about one warp per scheduler, waited
// on those chains (1.9 M cycles a permutation).  With 29-bit limbs a product
// column (at most 45 + 9 products below 2^58) fits 64 bits, so the columns are
// plain 64-bit multiply-adds, independent of each other; carries are taken
// once per column of the Montgomery reduction.  171 wide multiply-adds against
// 136, no carry flags, and a squaring takes 135.  Forests: 2^14 x 135 18.1 ->
// 14.6 ms, 2^18 x 32 37.8 -> 29.5 ms.  (The same 32-bit limbs summed in even
// and odd pairs as hand-written carry chains: 25.1 and 46.2 ms.)
//
// Values are x R mod r, R = 2^261, any representative below 2^261 (169 r) with
// limbs below 2^29: a product of representatives below a r and b r is below
// (a b / 169 + 1) r, so nothing is reduced further until the permutation's
// end.  Inside it no value exceeds 90 r: slots 1..4 gain less than 1.5 r in
// each of the 60 partial rounds, every other value is below 45 r.
#pragma once
#include <stdint.h>

#include "gl64.cuh"
#include "mma_tables.inc"

namespace zk {

#ifdef __CUDACC__

static __constant__ uint32_t d_FR29[ZK_FR29_WORDS] = {ZK_FR29_LIST};  // C, S, M, P, R^2 mod r (element order of zk_constants.h)
enum : int { FR29_C = 0, FR29_S = 100, FR29_M = 640, FR29_P = 665, FR29_R2 = 690 };

struct Fr29 {
    uint32_t w[9];
};

static constexpr uint32_t FR29_MASK = (1u << 29) - 1;

__host__ __device__ constexpr uint32_t fr29_r(int i)
{
    constexpr uint32_t r[9] = {ZK_FR29_R_LIST};
    return r[i];
}

__device__ __forceinline__ Fr29 fr29_const(int idx)
{
    Fr29 z;
#pragma unroll
    for (int k = 0; k < 9; k++) z.w[k] = d_FR29[9 * idx + k];
    return z;
}

// carries moved up: limbs below 2^29 again (the value is below 2^261)
__device__ __forceinline__ void fr29_carry(Fr29 &a)
{
#pragma unroll
    for (int k = 0; k < 8; k++) {
        a.w[k + 1] += a.w[k] >> 29;
        a.w[k] &= FR29_MASK;
    }
}

__device__ __forceinline__ Fr29 fr29_add(const Fr29 &a, const Fr29 &b)
{
    Fr29 z;
#pragma unroll
    for (int k = 0; k < 9; k++) z.w[k] = a.w[k] + b.w[k];
    fr29_carry(z);
    return z;
}

__device__ __forceinline__ void fr29_columns_add(uint64_t c[17], const Fr29 &a, const Fr29 &b)
{
#pragma unroll
    for (int i = 0; i < 9; i++)
#pragma unroll
        for (int j = 0; j < 9; j++) c[i + j] += (uint64_t)a.w[i] * b.w[j];
}

// (sum of columns) / R mod r.  Column k's m makes it vanish mod 2^29.
__device__ __forceinline__ Fr29 fr29_montgomery(uint64_t c[17])
{
#pragma unroll
    for (int k = 0; k < 9; k++) {
        const uint32_t m = ((uint32_t)c[k] * ZK_FR29_NP) & FR29_MASK;
#pragma unroll
        for (int j = 0; j < 9; j++) c[k + j] += (uint64_t)m * fr29_r(j);
        c[k + 1] += c[k] >> 29;
    }
    Fr29 z;
#pragma unroll
    for (int k = 9; k < 17; k++) {
        z.w[k - 9] = (uint32_t)c[k] & FR29_MASK;
        if (k < 16) c[k + 1] += c[k] >> 29;
    }
    z.w[8] = (uint32_t)(c[16] >> 29);
    return z;
}

// Out of line: one copy each of the code a permutation runs about 600 times.
static __device__ __noinline__ Fr29 fr29_mul(const Fr29 a, const Fr29 b)
{
    uint64_t c[17] = {};
    fr29_columns_add(c, a, b);
    return fr29_montgomery(c);
}

static __device__ __noinline__ Fr29 fr29_sqr(const Fr29 a)
{
    uint64_t c[17] = {};
#pragma unroll
    for (int i = 0; i < 9; i++) {
        c[2 * i] += (uint64_t)a.w[i] * a.w[i];
        const uint32_t d = 2 * a.w[i];
#pragma unroll
        for (int j = i + 1; j < 9; j++) c[i + j] += (uint64_t)d * a.w[j];
    }
    return fr29_montgomery(c);
}

// sum_j constant(c0 + j * step) * s_j, reduced once (45 + 9 products a column)
static __device__ __noinline__ Fr29 fr29_dot5(int c0, int step, const Fr29 s0, const Fr29 s1, const Fr29 s2, const Fr29 s3,
                                              const Fr29 s4)
{
    uint64_t c[17] = {};
    fr29_columns_add(c, s0, fr29_const(c0));
    fr29_columns_add(c, s1, fr29_const(c0 + step));
    fr29_columns_add(c, s2, fr29_const(c0 + 2 * step));
    fr29_columns_add(c, s3, fr29_const(c0 + 3 * step));
    fr29_columns_add(c, s4, fr29_const(c0 + 4 * step));
    return fr29_montgomery(c);
}

__device__ __forceinline__ Fr29 fr29_exp5(const Fr29 &x) { return fr29_mul(fr29_sqr(fr29_sqr(x)), x); }

// Out of Montgomery form, canonical, the low 192 bits as three lanes (most
// significant word first), each reduced once mod p.
__device__ __forceinline__ void fr29_words(const Fr29 &x, uint64_t s[3])
{
    Fr29 one;
#pragma unroll
    for (int k = 0; k < 9; k++) one.w[k] = k == 0;
    const Fr29 v = fr29_mul(x, one);  // at most r
    Fr29 d;                           // v - r when v >= r
    uint32_t borrow = 0;
#pragma unroll
    for (int k = 0; k < 9; k++) {
        const uint32_t t = v.w[k] - fr29_r(k) - borrow;
        borrow = t >> 31;
        d.w[k] = t & FR29_MASK;
    }
#pragma unroll
    for (int k = 0; k < 9; k++) d.w[k] = borrow ? v.w[k] : d.w[k];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        uint64_t limb = 0;
#pragma unroll
        for (int j = 0; j < 9; j++) {
            const int at = 29 * j - 64 * k;  // limb j's first bit in this word
            if (at > -29 && at < 0) limb |= (uint64_t)d.w[j] >> -at;
            else if (at >= 0 && at < 64) limb |= (uint64_t)d.w[j] << at;
        }
        s[2 - k] = gl_canon(limb);
    }
}

// poseidon_bn128_permute (hash.cuh) on the 12 Goldilocks lanes.
__device__ __forceinline__ void poseidon_bn128_permute29(uint64_t s[12])
{
    Fr29 st[5];
#pragma unroll
    for (int k = 0; k < 9; k++) st[0].w[k] = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint64_t l[3] = {gl_canon(s[3 * i + 2]), gl_canon(s[3 * i + 1]), gl_canon(s[3 * i])};
        Fr29 x;
#pragma unroll
        for (int k = 0; k < 9; k++) {
            const int bit = 29 * k, q = bit >> 6, sh = bit & 63;
            uint64_t v = q < 3 ? l[q] >> sh : 0;
            if (sh > 35 && q + 1 < 3) v |= l[q + 1] << (64 - sh);
            x.w[k] = (uint32_t)v & FR29_MASK;
        }
        st[1 + i] = fr29_mul(x, fr29_const(FR29_R2));
    }
#pragma unroll
    for (int i = 0; i < 5; i++) st[i] = fr29_add(st[i], fr29_const(FR29_C + i));
#pragma unroll 1
    for (int f = 0; f < 8; f++) {
#pragma unroll
        for (int i = 0; i < 5; i++) st[i] = fr29_exp5(st[i]);
        if (f != 7) {
            const int c0 = FR29_C + (f < 4 ? 5 * (f + 1) : 85 + 5 * (f - 4));
#pragma unroll
            for (int i = 0; i < 5; i++) st[i] = fr29_add(st[i], fr29_const(c0 + i));
        }
        // new_i = sum_j m[j][i] s_j, shifted into place (one call site)
        Fr29 ns[5];
        const int m0 = f == 3 ? FR29_P : FR29_M;
#pragma unroll 1
        for (int i = 0; i < 5; i++) {
            const Fr29 o = fr29_dot5(m0 + i, 5, st[0], st[1], st[2], st[3], st[4]);
#pragma unroll
            for (int q = 0; q < 4; q++) ns[q] = ns[q + 1];
            ns[4] = o;
        }
#pragma unroll
        for (int i = 0; i < 5; i++) st[i] = ns[i];
        if (f == 3) {
#pragma unroll 1
            for (int r = 0; r < 60; r++) {
                const Fr29 x0 = fr29_add(fr29_exp5(st[0]), fr29_const(FR29_C + 25 + r));
                const Fr29 n0 = fr29_dot5(FR29_S + 9 * r, 1, x0, st[1], st[2], st[3], st[4]);
#pragma unroll
                for (int k = 1; k < 5; k++) st[k] = fr29_add(st[k], fr29_mul(x0, fr29_const(FR29_S + 9 * r + 4 + k)));
                st[0] = n0;
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; i++) fr29_words(st[i], s + 3 * i);
}

// ---- one state per five threads.  A permutation on one thread is about 1 M
// cycles, which the narrow levels of a tree and forests of a few thousand
// leaves wait on.  Here thread i < 5 of a group holds state slot i, six groups
// to a warp (threads 30 and 31 repeat a group that does not exist): the S-boxes
// of a full round run side by side, and of a partial round's products only the
// three of slot 0's S-box and one more are in sequence.  All 32 threads call
// together.
struct Fr29Group {
    uint32_t i, base;  // slot, first thread of the group
    bool live;
    __device__ __forceinline__ void init()
    {
        const uint32_t lane = threadIdx.x & 31u;
        i = lane % 5;
        base = lane - i;
        live = lane < 30;
    }
};

// constants read at another index by every thread: the constant bank would
// serialise them
static __device__ const uint32_t g_FR29[ZK_FR29_WORDS] = {ZK_FR29_LIST};

__device__ __forceinline__ Fr29 fr29_const_g(int idx)
{
    Fr29 z;
#pragma unroll
    for (int k = 0; k < 9; k++) z.w[k] = __ldg(&g_FR29[9 * idx + k]);
    return z;
}

// slot j's element, in every thread of the group
__device__ __forceinline__ Fr29 fr29_from(const Fr29 &a, const Fr29Group &g, uint32_t j)
{
    Fr29 z;
#pragma unroll
    for (int k = 0; k < 9; k++) z.w[k] = __shfl_sync(0xFFFFFFFFu, a.w[k], (g.base + j) & 31u);
    return z;
}

// s: lanes 3 (i - 1) .. 3 (i - 1) + 2 of the state in threads 1..4.  Bounds as
// above, but for slot 0 in the partial rounds: a sum of five reduced products,
// below 7 r.
__device__ __forceinline__ void poseidon_bn128_permute_group(uint64_t s[3], const Fr29Group &g)
{
    Fr29 st;
    {
        const uint64_t l[3] = {gl_canon(s[2]), gl_canon(s[1]), gl_canon(s[0])};
        Fr29 x;
#pragma unroll
        for (int k = 0; k < 9; k++) {
            const int bit = 29 * k, q = bit >> 6, sh = bit & 63;
            uint64_t v = q < 3 ? l[q] >> sh : 0;
            if (sh > 35 && q + 1 < 3) v |= l[q + 1] << (64 - sh);
            x.w[k] = g.i ? (uint32_t)v & FR29_MASK : 0;
        }
        st = fr29_add(fr29_mul(x, fr29_const_g(FR29_R2)), fr29_const_g(FR29_C + g.i));
    }
#pragma unroll 1
    for (int f = 0; f < 8; f++) {
        st = fr29_exp5(st);
        if (f != 7) st = fr29_add(st, fr29_const_g(FR29_C + (f < 4 ? 5 * (f + 1) : 85 + 5 * (f - 4)) + g.i));
        uint64_t c[17] = {};
        const int m0 = (f == 3 ? FR29_P : FR29_M) + g.i;
#pragma unroll 1
        for (int j = 0; j < 5; j++) fr29_columns_add(c, fr29_from(st, g, j), fr29_const_g(m0 + 5 * j));
        st = fr29_montgomery(c);
        if (f == 3) {
#pragma unroll 1
            for (int r = 0; r < 60; r++) {
                const int row = FR29_S + 9 * r;
                // slot 0 squares, the others take their term of its row
                const Fr29 sk = fr29_const_g(row + g.i);
                Fr29 b;
#pragma unroll
                for (int k = 0; k < 9; k++) b.w[k] = g.i ? sk.w[k] : st.w[k];
                const Fr29 p = fr29_mul(st, b);
                const Fr29 x5 = fr29_mul(fr29_sqr(p), st);
                const Fr29 x0 = fr29_from(fr29_add(x5, fr29_const_g(FR29_C + 25 + r)), g, 0);
                const Fr29 v = fr29_mul(x0, fr29_const_g(g.i ? row + 4 + g.i : row));
                const Fr29 next = fr29_add(st, v);  // slots 1..4
                Fr29 sum = v;                       // slot 0
#pragma unroll
                for (uint32_t j = 1; j < 5; j++) {
                    const Fr29 t = fr29_from(p, g, j);
#pragma unroll
                    for (int k = 0; k < 9; k++) sum.w[k] += t.w[k];
                }
                fr29_carry(sum);
#pragma unroll
                for (int k = 0; k < 9; k++) st.w[k] = g.i ? next.w[k] : sum.w[k];
            }
        }
    }
    // slots 0..3 go to the elements of threads 1..4
    st = fr29_from(st, g, (g.i + 4) % 5);
    fr29_words(st, s);
}

// Plonky2's sponge (hash.cuh sponge_hash_one) with the state in the group; all
// threads of a group pass the same src and len > 4.  Digest words 0..2 are left
// in thread 1's out, word 3 in thread 2's out[0].
__device__ __forceinline__ void sponge_bn128_group(const uint64_t *src, uint64_t len, uint64_t out[3], const Fr29Group &g)
{
    out[0] = out[1] = out[2] = 0;
    const uint32_t l0 = g.i ? 3 * (g.i - 1) : 12;  // this thread's first lane
#pragma unroll 1
    for (uint64_t idx = 0; idx < len; idx += 8) {
#pragma unroll
        for (uint32_t q = 0; q < 3; q++)
            if (l0 + q < 8 && idx + l0 + q < len) out[q] = src[idx + l0 + q];
        poseidon_bn128_permute_group(out, g);
    }
}

#endif  // __CUDACC__

}  // namespace zk
