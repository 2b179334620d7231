// hash_mma.cuh -- Poseidon, Poseidon2 and Monolith with their linear layers on the
// tensor cores (8-bit products, 32-bit sums, exact), one warp for up to 32
// states.
//
// What bounds the one-thread-per-state form (hash.cuh) is issue on the integer
// pipes: of a permutation's ~20 K (Poseidon2) to ~26 K (Poseidon) instructions
// more than half are linear layers.  Here those are byte-matrix products with
// the tables of mma_tables.h: eight 32-bit sums per output lane, recombined in
// about 15 instructions whatever the number of input lanes, so what is left is
// the S-boxes.
//
// Layout.  A quad of threads (t = lane & 3) holds NS = 4 states (two 16-row
// tiles x rows g and g + 8, g = lane >> 2), 2 (one tile) or 1 (its row g); thread t
// has lanes t, 4 + t and 8 + t of each.  A lane's two 32-bit halves are the
// thread's A operand as they stand, and the columns of the tables are ordered
// so that thread t receives all byte sums of its own output lanes: a full
// round exchanges nothing between threads.  In the partial rounds the four
// values of a block of four rounds go to one thread per state through shared
// memory (thread t takes state t mod NS; for NS < 4 several threads repeat
// a state's chain), which runs the four S-boxes in sequence; their outputs
// become the A operand of the next k-block the same way.
#pragma once
#include <stdint.h>

#include "hash.cuh"
#include "mma_layout.h"
#include "mma_tables.inc"

namespace zk {

#ifdef __CUDACC__

template <int H>
struct HasMma {
    static constexpr bool value = H == HASH_POSEIDON || H == HASH_POSEIDON2 || H == HASH_MONOLITH;
};

static __device__ const __align__(16) uint32_t g_mma_poseidon[MMA_WORDS] = {ZK_MMA_POSEIDON_LIST};
static __device__ const __align__(16) uint32_t g_mma_poseidon2[MMA_WORDS] = {ZK_MMA_POSEIDON2_LIST};
static __device__ const __align__(16) uint32_t g_mma_monolith[MMA_MONO_WORDS] = {ZK_MMA_MONOLITH_LIST};

static __device__ const uint64_t g_mma_rc0[12] = {ZK_MMA_POSEIDON_RC0};  // Poseidon's first constants

template <int H>
constexpr uint32_t mma_table_words() { return H == HASH_MONOLITH ? MMA_MONO_WORDS : MMA_WORDS; }

template <int H>
__device__ __forceinline__ const uint32_t *mma_table()
{
    if constexpr (H == HASH_POSEIDON) return g_mma_poseidon;
    else if constexpr (H == HASH_POSEIDON2) return g_mma_poseidon2;
    else return g_mma_monolith;
}

// Shared-memory words (32-bit) one warp needs: the A operands [k-block 9][tile]
// [thread][4 or 2] (the 12 lanes entering a layer and the 22 S-box outputs of
// the partial rounds).  The exchange of a block of partial rounds, [quad 8]
// [state 4 ^ (quad & 3)][value 4] of 64 bits (the order of the states keeps its
// accesses free of bank conflicts), goes through the k-block that its S-box
// outputs fill afterwards.
template <int NS>
struct MmaSmem {
    static constexpr int TILES = NS == 4 ? 2 : 1, ROWS = NS == 1 ? 1 : 2;
    static constexpr int TILE = 32 * 2 * ROWS, BLOCK = TILES * TILE;
    static constexpr int XCHG = 8 * 4 * 4 * 2;
    // groups of output lanes worked on side by side: one and two states per
    // quad are the latency forms, whose S-boxes of a round run interleaved
    static constexpr int GROUPS = NS == 4 ? 1 : 3;
    static constexpr int WORDS = 8 * BLOCK + (XCHG > BLOCK ? XCHG : BLOCK);
    // Monolith has no partial rounds: its 12 lanes alone
    template <int H>
    static constexpr int words() { return H == HASH_MONOLITH ? 3 * BLOCK : WORDS; }
};

__device__ __forceinline__ void mma_16832(uint32_t d[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                          uint32_t b1, const uint32_t c[4])
{
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %11, %12, %13};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(c[0]), "r"(c[1]), "r"(c[2]), "r"(c[3]));
}

// s0 + 2^8 s1 + ... + 2^56 s7 as a 64-bit representative.  257 times the
// largest sum is below 2^32 (mma_sums_fit, checked when the tables are made).
__device__ __forceinline__ uint64_t mma_combine(uint32_t s0, uint32_t s1, uint32_t s2, uint32_t s3, uint32_t s4,
                                                uint32_t s5, uint32_t s6, uint32_t s7)
{
    const uint32_t u0 = s0 + s1 * 256u, u1 = s2 + s3 * 256u, u2 = s4 + s5 * 256u, u3 = s6 + s7 * 256u;
    uint32_t t0, t1;
    asm("{\n\t"
        ".reg .u64 a, b;\n\t"
        ".reg .u32 a0, a1, b0, b1, c;\n\t"
        "mul.wide.u32    a, %3, 65536;\n\t"
        "mul.wide.u32    b, %5, 65536;\n\t"
        "mov.b64         {a0, a1}, a;\n\t"
        "mov.b64         {b0, b1}, b;\n\t"
        "add.cc.u32      b0, b0, %4;\n\t"   // r = u0 + 2^16 u1 + 2^32 u2 + 2^48 u3 = {%1, %0} + 2^64 b1, b1 < 2^17
        "addc.u32        b1, b1, 0;\n\t"
        "add.cc.u32      %0, a0, %2;\n\t"
        "addc.cc.u32     %1, a1, b0;\n\t"
        "addc.u32        b1, b1, 0;\n\t"
        "mad.lo.cc.u32   %0, b1, 0xffffffff, %0;\n\t"  // + b1 * EPS, one EPS more on a carry
        "madc.hi.cc.u32  %1, b1, 0xffffffff, %1;\n\t"
        "addc.u32        c, 0, 0;\n\t"
        "neg.s32         c, c;\n\t"
        "add.cc.u32      %0, %0, c;\n\t"
        "addc.u32        %1, %1, 0;\n\t"
        "}"
        : "=&r"(t0), "=&r"(t1)
        : "r"(u0), "r"(u1), "r"(u2), "r"(u3));
    return ((uint64_t)t1 << 32) | t0;
}

// One tile's operands of one k-block: for two rows {low q0, low q1, high q0,
// high q1} as one 16-byte access, the registers mma.sync reads.
template <int NS>
struct MmaA {
    uint32_t w[4];
    __device__ __forceinline__ void load(const uint32_t *p)
    {
        if constexpr (MmaSmem<NS>::ROWS == 2) {
            const uint4 v = *(const uint4 *)p;
            w[0] = v.x;
            w[1] = v.y;
            w[2] = v.z;
            w[3] = v.w;
        } else {
            const uint2 v = *(const uint2 *)p;
            w[0] = v.x;
            w[1] = w[3] = 0;
            w[2] = v.y;
        }
    }
    static __device__ __forceinline__ void store(uint32_t *p, const uint64_t *x)
    {
        if constexpr (MmaSmem<NS>::ROWS == 2)
            *(uint4 *)p = make_uint4((uint32_t)x[0], (uint32_t)x[1], (uint32_t)(x[0] >> 32), (uint32_t)(x[1] >> 32));
        else
            *(uint2 *)p = make_uint2((uint32_t)x[0], (uint32_t)(x[0] >> 32));
    }
    __device__ __forceinline__ uint64_t row(int r) const { return ((uint64_t)w[2 + r] << 32) | w[r]; }
};

// A group's lanes (k-block) back into sm.
template <int NS>
__device__ __forceinline__ void mma_store_group(uint32_t *p, const uint64_t *v)
{
    using M = MmaSmem<NS>;
#pragma unroll
    for (int k = 0; k < M::TILES; k++) MmaA<NS>::store(p + k * M::TILE, v + M::ROWS * k);
}

// Table words through L1, or from a copy in shared memory (TSM).
template <bool TSM>
__device__ __forceinline__ uint4 mma_ld(const uint32_t *p)
{
    if constexpr (TSM) return *(const uint4 *)p;
    else return __ldg((const uint4 *)p);
}

// Sums of one group of four output lanes.
template <int NS, bool TSM>
struct MmaAcc {
    using M = MmaSmem<NS>;
    uint32_t s[M::TILES][4][4];
    __device__ __forceinline__ void start(const uint32_t *c)
    {
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const uint4 v = mma_ld<TSM>(c + 16 * i);
#pragma unroll
            for (int k = 0; k < M::TILES; k++) {
                s[k][i][0] = v.x;
                s[k][i][1] = v.y;
                s[k][i][2] = v.z;
                s[k][i][3] = v.w;
            }
        }
    }
    __device__ __forceinline__ void add(const MmaA<NS> *a, const uint32_t *b)
    {
        const uint4 p = mma_ld<TSM>(b), q = mma_ld<TSM>(b + 128);
#pragma unroll
        for (int k = 0; k < M::TILES; k++) {
            const uint32_t *w = a[k].w;
            mma_16832(s[k][0], w[0], w[1], w[2], w[3], p.x, p.y, s[k][0]);
            mma_16832(s[k][1], w[0], w[1], w[2], w[3], p.z, p.w, s[k][1]);
            mma_16832(s[k][2], w[0], w[1], w[2], w[3], q.x, q.y, s[k][2]);
            mma_16832(s[k][3], w[0], w[1], w[2], w[3], q.z, q.w, s[k][3]);
        }
    }
    // += a full-round layer (mma_full_operands)
    __device__ __forceinline__ void add_full(const uint32_t (*a)[4][4], const uint32_t *b)
    {
        const uint4 p = mma_ld<TSM>(b), q = mma_ld<TSM>(b + 128);
#pragma unroll
        for (int k = 0; k < M::TILES; k++) {
            mma_16832(s[k][0], a[k][0][0], a[k][0][1], a[k][0][2], a[k][0][3], p.x, p.y, s[k][0]);
            mma_16832(s[k][1], a[k][1][0], a[k][1][1], a[k][1][2], a[k][1][3], p.z, p.w, s[k][1]);
            mma_16832(s[k][2], a[k][2][0], a[k][2][1], a[k][2][2], a[k][2][3], q.x, q.y, s[k][2]);
            mma_16832(s[k][3], a[k][3][0], a[k][3][1], a[k][3][2], a[k][3][3], q.z, q.w, s[k][3]);
        }
    }
    __device__ __forceinline__ void add_smem(const uint32_t *a, const uint32_t *b)
    {
        MmaA<NS> x[M::TILES];
#pragma unroll
        for (int k = 0; k < M::TILES; k++) x[k].load(a + k * M::TILE);
        add(x, b);
    }
    __device__ __forceinline__ void finish(uint64_t out[NS]) const
    {
#pragma unroll
        for (int q = 0; q < NS; q++) {
            const auto &v = s[q / M::ROWS];
            const int r = 2 * (q % M::ROWS);
            out[q] = mma_combine(v[0][r], v[0][r + 1], v[1][r], v[1][r + 1], v[2][r], v[2][r + 1], v[3][r], v[3][r + 1]);
        }
    }
};

// The coefficients inside a block of partial rounds applied: y + sum_d h_d x_(-d).
template <int H, int N>
__device__ __forceinline__ uint64_t mma_chain(uint64_t y, const uint64_t x[3])
{
    if constexpr (H == HASH_POSEIDON) {
        constexpr uint32_t h[3] = {(uint32_t)ZK_MMA_POSEIDON_H1, (uint32_t)ZK_MMA_POSEIDON_H2, (uint32_t)ZK_MMA_POSEIDON_H3};
        static_assert(ZK_MMA_POSEIDON_H3 < (1ULL << 22), "coefficients of one word");
        Acc96 a;
        a.lo = (uint32_t)y;
        a.hi = y >> 32;
#pragma unroll
        for (int d = 0; d < N; d++) a.mac(x[N - 1 - d], h[d]);
        return a.reduce();
    } else {
        constexpr uint64_t h[3] = {ZK_MMA_POSEIDON2_H1, ZK_MMA_POSEIDON2_H2, ZK_MMA_POSEIDON2_H3};
        static_assert(ZK_MMA_POSEIDON2_H2 == 11, "lane 0 comes back through the other eleven lanes");
        if constexpr (N == 1) return gl_mul_add_nc(x[0], h[0], y);
        else if constexpr (N == 2) {
            Acc96 a;
            a.lo = (uint32_t)y;
            a.hi = y >> 32;
            a.mac(x[0], (uint32_t)h[1]);
            return gl_mul_add_nc(x[1], h[0], a.reduce());
        } else {
            Acc96 a;
            a.lo = (uint32_t)y;
            a.hi = y >> 32;
            a.mac(x[1], (uint32_t)h[1]);
            WideAcc w;
            w.start(a.reduce());
            w.mac(x[2], h[0]);
            w.mac(x[0], h[2]);
            return w.reduce();
        }
    }
}

// Operands of a full-round layer from the state at a.  Its coefficients are
// below 256, so byte b of an output takes byte b of the lanes alone: for column
// pair i one k-block with bytes 2i and 2i + 1 of lanes t and 4 + t and the word
// of lane 8 + t that has them, a third of the products of the byte matrix.
template <int NS>
__device__ __forceinline__ void mma_full_operands(uint32_t (*x)[4][4], const uint32_t *a)
{
    using M = MmaSmem<NS>;
#pragma unroll
    for (int k = 0; k < M::TILES; k++) {
        MmaA<NS> y[3];
#pragma unroll
        for (int kb = 0; kb < 3; kb++) y[kb].load(a + kb * M::BLOCK + k * M::TILE);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int h = 2 * (i >> 1);
            const uint32_t sel = i & 1 ? 0x7632 : 0x5410;
#pragma unroll
            for (int r = 0; r < 2; r++) {
                x[k][i][r] = r < M::ROWS ? __byte_perm(y[0].w[h + r], y[1].w[h + r], sel) : 0;
                x[k][i][2 + r] = y[2].w[h + r];
            }
        }
    }
}

// Block i < 6 of the partial rounds (four rounds, two in the last): 3 + i
// k-blocks of operands, the S-box outputs into k-block 3 + i.
template <int H, int NS, bool TSM>
__device__ __forceinline__ void mma_rounds4(uint32_t *sm, const uint32_t *b, const uint32_t *c, int i)
{
    using M = MmaSmem<NS>;
    const uint32_t lane = threadIdx.x & 31, t = lane & 3, g = lane >> 2;
    const uint32_t q = t % NS;  // the state whose S-box chain this thread runs
    const uint32_t *a = sm + lane * 2 * M::ROWS;
    MmaAcc<NS, TSM> acc;
    acc.start(c);
#pragma unroll
    for (int kb = 0; kb < 3; kb++) acc.add_smem(a + kb * M::BLOCK, b + kb * MMA_KB);
#pragma unroll 1
    for (int kb = 3; kb < 3 + i; kb++) acc.add_smem(a + kb * M::BLOCK, b + kb * MMA_KB);
    uint32_t *xo = sm + (3 + i) * M::BLOCK;
    uint64_t *xc = (uint64_t *)xo + 16 * g;
    uint64_t x[4];
    acc.finish(x);
#pragma unroll
    for (int k = 0; k < NS; k++) xc[4 * (k ^ (g & 3)) + t] = x[k];
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 4; j += 2) {
        const ulonglong2 v = *(const ulonglong2 *)(xc + 4 * (q ^ (g & 3)) + j);
        x[j] = v.x;
        x[j + 1] = v.y;
    }
    __syncwarp();
    x[0] = gl_sbox7_nc(x[0]);
    x[1] = gl_sbox7_nc(mma_chain<H, 1>(x[1], x));
    if (i < 5) {  // else the coefficients of x_2 and x_3 are zero
        x[2] = gl_sbox7_nc(mma_chain<H, 2>(x[2], x));
        x[3] = gl_sbox7_nc(mma_chain<H, 3>(x[3], x));
    }
    if (t < NS) {
        // x_j is the operand of thread j of the quad
        uint32_t *xw = xo + (q / M::ROWS) * M::TILE + 4 * g * 2 * M::ROWS + q % M::ROWS;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            xw[j * 2 * M::ROWS] = (uint32_t)x[j];
            xw[j * 2 * M::ROWS + M::ROWS] = (uint32_t)(x[j] >> 32);
        }
    }
    __syncwarp();
}

// One permutation of the warp's states, in place in sm (k-block kb: lanes
// 4 kb + t).  Bit j of `groups`: lanes 4j..4j+3 of the result are needed (the
// others keep values of no meaning): a sponge needs lanes 8..11 between full
// chunks and lanes 0..3 at its end.  Every thread of the warp calls together;
// groups is the same in all of them.
//
// One rolled loop over the layers, each a rolled loop over three groups of
// output lanes (product, recombination, S-boxes, store), so that the whole
// permutation is ~1300 instructions: unrolled forms of ~3000 stalled on
// instruction fetch.  A layer reads its operands into registers before its
// first store, and a thread's slots are its own, so it works in place.
template <int H, int NS, bool TSM = false>
__device__ __forceinline__ void permute_mma(uint32_t *sm, uint32_t groups, const uint32_t *table = mma_table<H>())
{
    using M = MmaSmem<NS>;
    const uint32_t lane = threadIdx.x & 31, t = lane & 3;
    constexpr int J = MmaSmem<NS>::GROUPS;
    uint32_t *a = sm + lane * 2 * M::ROWS;
    const uint32_t *tab = table + 4 * lane, *cst = table + 4 * t;
#pragma unroll 1
    for (int st = 0; st < 10; st++) {
        if (st == 4) {  // the partial rounds
            const uint32_t *b = tab + MMA_Y, *c = cst + MMA_YCONST;
#pragma unroll 1
            for (int i = 0; i < 6; i++, c += MMA_GROUP) {
                mma_rounds4<H, NS, TSM>(sm, b, c, i);
                b += (3 + i) * MMA_KB;
            }
            b = tab + MMA_W;
            c = cst + MMA_CONST + 12 * MMA_GROUP;
            MmaA<NS> x[3][M::TILES];
#pragma unroll
            for (int kb = 0; kb < 3; kb++)
#pragma unroll
                for (int k = 0; k < M::TILES; k++) x[kb][k].load(a + kb * M::BLOCK + k * M::TILE);
#pragma unroll 1
            for (int j0 = 0; j0 < 3; j0 += J, b += 9 * J * MMA_KB, c += J * MMA_GROUP) {
                MmaAcc<NS, TSM> acc[J];
#pragma unroll
                for (int j = 0; j < J; j++) {
                    acc[j].start(c + j * MMA_GROUP);
#pragma unroll
                    for (int kb = 0; kb < 3; kb++) acc[j].add(x[kb], b + (9 * j + kb) * MMA_KB);
                }
#pragma unroll 2
                for (int kb = 3; kb < 9; kb++)
#pragma unroll
                    for (int j = 0; j < J; j++) acc[j].add_smem(a + kb * M::BLOCK, b + (9 * j + kb) * MMA_KB);
#pragma unroll
                for (int j = 0; j < J; j++) {
                    uint64_t v[NS];
                    acc[j].finish(v);
                    mma_store_group<NS>(a + (j0 + j) * M::BLOCK, v);
                }
            }
            continue;
        }
        const bool raw = st == 5 || (H == HASH_POSEIDON && st == 0);  // S-boxes alone
        const uint32_t mask = st == 9 ? groups : 7u;
        const uint32_t *b = tab + MMA_FULL, *c = cst + MMA_CONST + 3 * MMA_GROUP * (st < 4 ? st : st - 1);
        uint32_t x[M::TILES][4][4];
        mma_full_operands<NS>(x, a);
#pragma unroll 1
        for (int j0 = 0; j0 < 3; j0 += J, b += J * MMA_KB, c += J * MMA_GROUP) {
            if (J == 1 && !((mask >> j0) & 1u)) continue;
            uint64_t v[J][NS];
            if (raw) {
#pragma unroll
                for (int j = 0; j < J; j++) {
                    const uint64_t rc = st ? 0 : __ldg(&g_mma_rc0[4 * (j0 + j) + t]);
#pragma unroll
                    for (int k = 0; k < M::TILES; k++) {
                        MmaA<NS> y;
                        y.load(a + (j0 + j) * M::BLOCK + k * M::TILE);
#pragma unroll
                        for (int r = 0; r < M::ROWS; r++) v[j][k * M::ROWS + r] = gl_add_nc(y.row(r), rc);
                    }
                }
            } else {
                MmaAcc<NS, TSM> acc[J];
#pragma unroll
                for (int j = 0; j < J; j++) {
                    acc[j].start(c + j * MMA_GROUP);
                    acc[j].add_full(x, b + j * MMA_KB);
                }
#pragma unroll
                for (int j = 0; j < J; j++) acc[j].finish(v[j]);
            }
            if (st != 9) {
#pragma unroll
                for (int q = 0; q < NS; q++)
#pragma unroll
                    for (int j = 0; j < J; j++) v[j][q] = gl_sbox7_nc(v[j][q]);
            }
#pragma unroll
            for (int j = 0; j < J; j++) mma_store_group<NS>(a + (j0 + j) * M::BLOCK, v[j]);
        }
    }
}

// a + b for any 64-bit a, b: the carry folded back as EPS, twice (the second
// time only when both operands are >= p).
__device__ __forceinline__ uint64_t mma_add_nc(uint64_t a, uint64_t b)
{
    uint32_t r0, r1, c;
    asm("{\n\t"
        "add.cc.u32      %0, %3, %5;\n\t"
        "addc.cc.u32     %1, %4, %6;\n\t"
        "addc.u32        %2, 0, 0;\n\t"
        "neg.s32         %2, %2;\n\t"
        "add.cc.u32      %0, %0, %2;\n\t"
        "addc.cc.u32     %1, %1, 0;\n\t"
        "addc.u32        %2, 0, 0;\n\t"
        "neg.s32         %2, %2;\n\t"
        "add.cc.u32      %0, %0, %2;\n\t"
        "addc.u32        %1, %1, 0;\n\t"
        "}"
        : "=&r"(r0), "=&r"(r1), "=&r"(c)
        : "r"((uint32_t)a), "r"((uint32_t)(a >> 32)), "r"((uint32_t)b), "r"((uint32_t)(b >> 32)));
    return ((uint64_t)r1 << 32) | r0;
}

// Monolith in the same form: Concrete (row 0), then six rounds of Bars on
// lanes 0..3, Bricks and Concrete.  Group 0 of a layer's output lanes is the
// one the Bars act on, one lane per thread; Bricks take the square of lane
// i - 1 from the thread before in the quad, or, for t = 0, the square of the
// group before from thread 3.
template <int NS, bool TSM = false>
__device__ __forceinline__ void permute_mma_monolith(uint32_t *sm, uint32_t groups, const uint32_t *table = g_mma_monolith)
{
    using M = MmaSmem<NS>;
    constexpr int J = M::GROUPS;
    const uint32_t lane = threadIdx.x & 31, t = lane & 3;
    uint32_t *a = sm + lane * 2 * M::ROWS;
    const uint32_t from = (lane & ~3u) | ((t + 3) & 3);
#pragma unroll 1
    for (int st = 0; st < 7; st++) {
        const uint32_t mask = st == 6 ? groups : 7u;
        const uint32_t *b = table + MMA_FULL + 4 * lane;
        const uint32_t *c = table + MMA_MONO_CONST + 3 * MMA_GROUP * st + 4 * t;
        uint32_t x[M::TILES][4][4];
        mma_full_operands<NS>(x, a);
        uint64_t prev[NS];  // squares of the group before
#pragma unroll
        for (int q = 0; q < NS; q++) prev[q] = 0;
#pragma unroll 1
        for (int j0 = 0; j0 < 3; j0 += J, b += J * MMA_KB, c += J * MMA_GROUP) {
            if (J == 1 && !((mask >> j0) & 1u)) continue;
            MmaAcc<NS, TSM> acc[J];
            uint64_t v[J][NS];
#pragma unroll
            for (int j = 0; j < J; j++) {
                acc[j].start(c + j * MMA_GROUP);
                acc[j].add_full(x, b + j * MMA_KB);
            }
#pragma unroll
            for (int j = 0; j < J; j++) acc[j].finish(v[j]);
            if (st < 6) {
                if (j0 == 0) {
#pragma unroll
                    for (int q = 0; q < NS; q++) v[0][q] = mono_bar(gl_canon(v[0][q]));
                }
#pragma unroll
                for (int j = 0; j < J; j++)
#pragma unroll
                    for (int q = 0; q < NS; q++) {
                        const uint64_t sq = gl_mul_nc(v[j][q], v[j][q]), send = t == 3 ? prev[q] : sq;
                        const uint32_t lo = __shfl_sync(0xFFFFFFFFu, (uint32_t)send, from);
                        const uint32_t hi = __shfl_sync(0xFFFFFFFFu, (uint32_t)(send >> 32), from);
                        prev[q] = sq;
                        v[j][q] = mma_add_nc(v[j][q], ((uint64_t)hi << 32) | lo);
                    }
            }
#pragma unroll
            for (int j = 0; j < J; j++) mma_store_group<NS>(a + (j0 + j) * M::BLOCK, v[j]);
        }
    }
}

// A state word of this thread (k-block kb, state q) in sm.
template <int NS>
__device__ __forceinline__ uint64_t mma_lane(const uint32_t *sm, int kb, int q)
{
    using M = MmaSmem<NS>;
    MmaA<NS> y;
    y.load(sm + kb * M::BLOCK + (q / M::ROWS) * M::TILE + (threadIdx.x & 31) * 2 * M::ROWS);
    return y.row(q % M::ROWS);
}

template <int NS>
__device__ __forceinline__ void mma_set_lane(uint32_t *sm, int kb, int q, uint64_t v)
{
    using M = MmaSmem<NS>;
    uint32_t *p = sm + kb * M::BLOCK + (q / M::ROWS) * M::TILE + (threadIdx.x & 31) * 2 * M::ROWS + q % M::ROWS;
    p[0] = (uint32_t)v;
    p[M::ROWS] = (uint32_t)(v >> 32);
}

// A word of a leaf or node row.  The 32-state form's rows are in global memory
// and read once, whole sectors at a time: kept out of L1, which the tables fill.
template <int NS>
__device__ __forceinline__ uint64_t mma_row_ld(const uint64_t *p)
{
    if constexpr (NS == 4) {
        uint64_t v;
        asm("ld.global.L1::no_allocate.u64 %0, [%1];" : "=l"(v) : "l"(p));
        return v;
    } else {
        return *p;
    }
}

// sponge_hash_one for the warp's states: row(q) is where state q's len words
// are; the digest word t of state q is left in d[q] (canonical).  len > 4.
template <int H, int NS, bool TSM = false, class Row>
__device__ __forceinline__ void sponge_hash_mma(Row row, uint64_t len, uint32_t *sm, uint64_t d[NS],
                                                const uint32_t *table = mma_table<H>())
{
    const uint32_t t = threadIdx.x & 3;
#pragma unroll
    for (int kb = 0; kb < 3; kb++)
#pragma unroll
        for (int q = 0; q < NS; q++) mma_set_lane<NS>(sm, kb, q, 0);
#pragma unroll 1
    for (uint64_t idx = 0; idx < len; idx += 8) {
#pragma unroll
        for (int q = 0; q < NS; q++) {
            const uint64_t *p = row(q) + idx;
            if (idx + t < len) mma_set_lane<NS>(sm, 0, q, mma_row_ld<NS>(p + t));
            if (idx + 4 + t < len) mma_set_lane<NS>(sm, 1, q, mma_row_ld<NS>(p + 4 + t));
        }
        // what the next chunk leaves in place: a full one lanes 8..11, one of
        // k < 8 words also lanes k..7
        const uint64_t rem = len - idx;
        const uint32_t groups = rem <= 8 ? 1u : rem >= 16 ? 4u : rem >= 12 ? 6u : 7u;
        if constexpr (H == HASH_MONOLITH) permute_mma_monolith<NS, TSM>(sm, groups, table);
        else permute_mma<H, NS, TSM>(sm, groups, table);
    }
#pragma unroll
    for (int q = 0; q < NS; q++) d[q] = gl_canon(mma_lane<NS>(sm, 0, q));
}

#endif  // __CUDACC__

}  // namespace zk
