// merkle.cu -- host driver of the Merkle forest builder.
//
// Follows native/merkle/merkle.cu:166-280 of zeknox for the layout and the
// special cases (caps == leaves; subtrees of 1 or 2 leaves).  Launches: the
// leaf kernel; one node-parallel level kernel per level while a level still
// has >= wide_level_nodes nodes; then folds inside CTAs.  Poseidon, Poseidon2
// and Monolith run their linear layers on the tensor cores (hash_mma.cuh), 32,
// 16 or 8 leaves per warp by the forest's size, and fold 6 levels per launch
// until a CTA holds whole subtrees; so does Poseidon-BN128, five threads a
// state in small forests and narrow levels.  Keccak hashes one leaf or node per
// thread: a fold kernel of 8 levels and, for subtrees still above 1024 nodes,
// level kernels, then one tail CTA per subtree.
#define ZK_BN128_LIMBS29 1
#include <algorithm>
#include <atomic>
#include <cstdio>
#include <string>

#include "geom.h"
#include "merkle.cuh"
#include "ntt_api.cuh"
#include "runtime.cuh"

namespace zk {

// Default threads per CTA of the leaf kernel ("leaf_threads.<hash>", 32 for
// the tensor-core hashes only).  Poseidon-BN128's holds 152 registers a
// thread: three 128-thread CTAs fit an SM where one 256-thread CTA does.  The
// tensor-core hashes take one-warp CTAs up to 2^16 leaves, where an SM has a
// handful of warps and larger CTAs leave some SMs one more than others
// (Poseidon2 2^15 x 135: 763 against 880 us with 64 threads and 640 a
// multiprocessor; 2^14: 493 against 509), above that 64 (Poseidon2
// 2^20 x 135: 14.11 against 14.18 ms) or, for Monolith, 128 (5.14 against 5.30).
static constexpr int LEAF_T = 256;
template <int H>
static uint64_t leaf_t_default(uint64_t n_leaves)
{
    if (H == HASH_POSEIDON_BN128) return 128;
    if (!HasMma<H>::value) return LEAF_T;
    return n_leaves <= (1ULL << 16) ? 32 : H == HASH_MONOLITH ? 128 : 64;
}
// Threads per CTA of the node-parallel level kernel: 128 for Poseidon-BN128
// (158 registers: three CTAs per SM instead of one), 256 otherwise.  The wide
// levels are ~6% of a forest's permutations: 2^20 x 135 Poseidon-BN128
// forest 449.0 against 450.2 ms.
template <int H>
constexpr unsigned level_t()
{
    return H == HASH_POSEIDON_BN128 ? 128u : 256u;
}
static constexpr int FOLD_T = 256;     // leaf digests per CTA of the fold kernel
static constexpr int TAIL_MAXM = 1024; // nodes a tail CTA can take
// Leaves per warp of the tensor-core leaf kernel: 8 up to coop_leaves leaves
// ("coop_leaves.<hash>"), 16 up to MID_LEAVES times as many, else 32.  Fewer
// per warp are fewer S-boxes in sequence and more warps, for more instructions
// a leaf.  Measured on B200, forests of 135-word leaves, 8 / 16 / 32 per warp
// (us): Poseidon 2^12 353 / 413 / 710, 2^14 652 / 499 / 708, 2^15 978 / 939 /
// 857; Poseidon2 the same within 5%; Monolith 2^12 108 / 128 / 214, 2^16
// 433 / 374 / 454, 2^17 800 / 679 / 740.
static constexpr uint64_t COOP_LEAVES = 1ULL << 12;
template <int H>
constexpr uint64_t mid_leaves()
{
    return H == HASH_MONOLITH ? 32 : 4;
}
static constexpr uint64_t WIDE_LEVEL_NODES = 1ULL << 15;  // default: levels at least this wide run node-parallel
                                                          // ("wide_level_nodes.<hash>")

// A level of a forest beside others counts their nodes too from this many of
// its own on (one batch of forests; not at all / from 1 / 2^9 / 2^11 / 2^13
// nodes, us, Poseidon2): 8 of 2^13 x 9 492 / 379 / 375 / 376 / 490; 2 of 2^18 and
// 14 of 2^9..2^12 x 8 1203 / 1419 / 1258 / 1161 / 1204; 64 of 2^10..2^16 x 8 5027 /
// 4062 / 3994 / 3943 / 4030; Poseidon alike, Monolith by less.
static constexpr uint64_t BESIDE_NODES = 1ULL << 11;

// Poseidon-BN128 forests up to this many leaves hash them with five threads a
// state ("coop_leaves.2"): 2^12 x 135 7.2 against 11.0 ms with one, 2^13 9.6
// against 11.2, 2^14 13.7 against 11.3.
static constexpr uint64_t BN128_COOP_LEAVES = 1ULL << 13;

bool merkle_geometry_ok(uint64_t n_digests, uint64_t n_caps, uint64_t n_leaves, uint64_t cap_height, std::string &err)
{
    return merkle_geometry_check(n_digests, n_caps, n_leaves, cap_height, err);
}

template <int H, int NS, int T>
static void launch_leaf_mma_t(uint64_t *digests, uint64_t *caps, const uint64_t *leaves, const MerkleGeom &g, cudaStream_t s)
{
    constexpr uint64_t per = (uint64_t)(T / 32) * 8 * NS;
    merkle_leaf_mma_kernel<H, NS, T><<<(unsigned)((g.n_leaves + per - 1) / per), T, 0, s>>>(leaves, digests, caps, g);
}

template <int H, int NS>
static void launch_leaf_mma(uint64_t lt, uint64_t *digests, uint64_t *caps, const uint64_t *leaves, const MerkleGeom &g,
                            cudaStream_t s)
{
    if (lt == 32) launch_leaf_mma_t<H, NS, 32>(digests, caps, leaves, g, s);
    else if (lt == 64) launch_leaf_mma_t<H, NS, 64>(digests, caps, leaves, g, s);
    else launch_leaf_mma_t<H, NS, 128>(digests, caps, leaves, g, s);
}

// Tables in shared memory while every CTA can have a multiprocessor to itself
// (forests of 8-word leaves, 2^10: Poseidon2 159 -> 147 us, Monolith 54 -> 47).
template <int H>
static void launch_fold_mma(unsigned ctas, uint64_t *digests, uint64_t *caps, const MerkleGeom &g, uint32_t u0, cudaStream_t s)
{
    constexpr uint32_t bytes = 4 * mma_table_words<H>();
    // the dynamic shared-memory opt-in is per device
    static std::atomic<uint64_t> attr_set{0};
    int dev = 0, sms = 0;
    bool copy = cudaGetDevice(&dev) == cudaSuccess &&
                cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && ctas <= (unsigned)sms;
    const uint64_t bit = 1ULL << (dev & 63);
    if (copy && !(attr_set.load(std::memory_order_relaxed) & bit)) {
        copy = cudaFuncSetAttribute(merkle_fold_mma_kernel<H, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)bytes) == cudaSuccess;
        if (copy) attr_set.fetch_or(bit, std::memory_order_relaxed);
        else (void)cudaGetLastError();  // the other form needs no opt-in
    }
    if (copy) merkle_fold_mma_kernel<H, true><<<ctas, 128, bytes, s>>>(digests, caps, g, u0);
    else merkle_fold_mma_kernel<H, false><<<ctas, 128, 0, s>>>(digests, caps, g, u0);
}

// One level, one node per thread, or 32 per warp.
template <int H>
static void launch_level(uint64_t total, uint64_t *digests, const MerkleGeom &g, uint32_t u, cudaStream_t s)
{
    if constexpr (HasMma<H>::value) {
        merkle_level_mma_kernel<H, 4, 128><<<(unsigned)((total + 127) / 128), 128, 0, s>>>(digests, g, u);
    } else {
        uint64_t nb = (total + level_t<H>() - 1) / level_t<H>();
        if (nb > 65535) nb = 65535;
        merkle_level_kernel<H><<<(unsigned)nb, level_t<H>(), 0, s>>>(digests, g, u);
    }
    note_launch();
}

// at_once: leaves of all forests that run at the same time, this one's among
// them.  Several forests' narrow levels fill the GPU together, where the
// fold's latency form (8 nodes per warp) costs more than one launch per level
// saves: a level is wide when the forests have wide_level_nodes nodes at its
// height between them.  Batches of Poseidon2 commits, each forest by its own
// width / by all of them (us): 7 of 2^13..2^15 leaves x 5..16 827 / 604, 9 of
// 2^12..2^16 x 8..20 1286 / 994.  The leaf kernel's form and the fold's
// table copy stay with the forest's own size: by all leaves the forms came out
// within 1% in the mean, and without the copy batches took 2% longer.
template <int H>
static void merkle_launch(uint64_t *digests, uint64_t *caps, const uint64_t *leaves, const MerkleGeom &g, uint64_t at_once,
                          cudaStream_t s)
{
    const uint32_t lg_leaves = ilog2_exact(g.n_leaves);
    const uint64_t lt = tune_get("leaf_threads." + std::to_string(H), lg_leaves, leaf_t_default<H>(g.n_leaves));
    uint64_t blocks;
    uint32_t u0 = 0;
    if constexpr (HasMma<H>::value) {
        const uint64_t coop =
            std::min<uint64_t>(tune_get("coop_leaves." + std::to_string(H), lg_leaves, COOP_LEAVES), 1ULL << 40);
        if (g.leaf_size <= 4) {
            blocks = (g.n_leaves + LEAF_T - 1) / LEAF_T;
            merkle_leaf_copy_kernel<LEAF_T><<<(unsigned)blocks, LEAF_T, 0, s>>>(leaves, digests, caps, g);
        } else if (g.n_leaves <= coop) {
            launch_leaf_mma<H, 1>(lt, digests, caps, leaves, g, s);
        } else if (g.n_leaves <= mid_leaves<H>() * coop) {
            launch_leaf_mma<H, 2>(lt, digests, caps, leaves, g, s);
        } else {
            launch_leaf_mma<H, 4>(lt, digests, caps, leaves, g, s);
        }
    } else if (H == HASH_POSEIDON_BN128 && g.leaf_size > 4 &&
               g.n_leaves <= tune_get("coop_leaves.2", lg_leaves, BN128_COOP_LEAVES)) {
        merkle_leaf_bn128_kernel<64><<<(unsigned)((g.n_leaves + 11) / 12), 64, 0, s>>>(leaves, digests, caps, g);
    } else if (lt == 64) {
        blocks = (g.n_leaves + 63) / 64;
        merkle_leaf_kernel<H, 64><<<(unsigned)blocks, 64, 0, s>>>(leaves, digests, caps, g);
    } else if (lt == 128) {
        blocks = (g.n_leaves + 127) / 128;
        merkle_leaf_kernel<H, 128><<<(unsigned)blocks, 128, 0, s>>>(leaves, digests, caps, g);
    } else {
        blocks = (g.n_leaves + LEAF_T - 1) / LEAF_T;
        merkle_leaf_kernel<H, LEAF_T><<<(unsigned)blocks, LEAF_T, 0, s>>>(leaves, digests, caps, g);
    }
    note_launch();
    const uint64_t wide = tune_get("wide_level_nodes." + std::to_string(H), lg_leaves, WIDE_LEVEL_NODES);
    if (g.sub_leaves == 1) return;  // caps == leaves
    // Wide levels: one node per thread while a level still fills the GPU.
    const uint32_t top = g.log_sub - 1;
    const auto wide_level = [&](uint32_t u) {
        const uint64_t nodes = g.n_leaves >> u;
        return nodes >= wide || (HasMma<H>::value && nodes >= BESIDE_NODES && (at_once >> u) >= wide);
    };
    while (u0 + 1 <= top && wide_level(u0 + 1)) {
        u0++;
        const uint64_t total = g.n_leaves >> u0;
        launch_level<H>(total, digests, g, u0, s);
    }
    // Narrow levels: folded inside CTAs of fold_nodes nodes; the tensor-core
    // form repeats until its CTAs hold whole subtrees.
    if constexpr (HasMma<H>::value || H == HASH_POSEIDON_BN128) {
        for (;;) {
            const uint64_t count = g.n_leaves >> u0;
            const unsigned ctas = (unsigned)((count + MMA_FOLD_IN - 1) / MMA_FOLD_IN);
            if constexpr (HasMma<H>::value) launch_fold_mma<H>(ctas, digests, caps, g, u0, s);
            else merkle_fold_bn128_kernel<<<ctas, 192, 0, s>>>(digests, caps, g, u0);
            note_launch();
            if ((g.sub_leaves >> u0) <= MMA_FOLD_IN) return;  // caps written
            u0 += __builtin_ctz(MMA_FOLD_IN);
        }
    } else {
        const uint64_t count = g.n_leaves >> u0;
        blocks = (count + FOLD_T - 1) / FOLD_T;
        merkle_fold_kernel<H, FOLD_T><<<(unsigned)blocks, FOLD_T, 0, s>>>(digests, caps, g, u0);
        note_launch();
        const uint64_t sub_nodes = g.sub_leaves >> u0;
        if (sub_nodes <= (uint64_t)FOLD_T) return;  // caps written by the fold kernel
        // heights folded by the fold kernel
        uint32_t U = 0;
        while ((1u << (U + 1)) <= FOLD_T && u0 + U + 1 <= top) U++;
        u0 += U;
        while ((g.sub_leaves >> u0) > (uint64_t)TAIL_MAXM) {
            u0++;
            launch_level<H>((g.sub_leaves >> u0) * g.n_caps, digests, g, u0, s);
        }
        merkle_tail_kernel<H, TAIL_MAXM><<<g.n_caps, 256, 0, s>>>(digests, caps, g, u0);
        note_launch();
    }
}

bool merkle_device(uint64_t *digests, uint64_t *caps, const uint64_t *leaves, uint64_t n_digests, uint64_t n_caps,
                   uint64_t n_leaves, uint64_t leaf_size, uint64_t cap_height, uint64_t hash_type, cudaStream_t stream,
                   std::string &err, uint64_t at_once)
{
    NvtxRange range("zeknox merkle");
    if (!merkle_geometry_ok(n_digests, n_caps, n_leaves, cap_height, err)) return false;
    if (n_caps > 0xFFFFFFFFULL) {
        err = "too many caps";
        return false;
    }
    MerkleGeom g;
    g.n_leaves = n_leaves;
    g.leaf_size = leaf_size;
    g.sub_leaves = n_leaves / n_caps;
    g.sub_digests = 2 * g.sub_leaves - 2;
    g.log_sub = ilog2_exact(g.sub_leaves);
    g.n_caps = (uint32_t)n_caps;
    switch (hash_type) {
    case HASH_POSEIDON: merkle_launch<HASH_POSEIDON>(digests, caps, leaves, g, at_once, stream); break;
    case HASH_KECCAK: merkle_launch<HASH_KECCAK>(digests, caps, leaves, g, at_once, stream); break;
    case HASH_POSEIDON_BN128: merkle_launch<HASH_POSEIDON_BN128>(digests, caps, leaves, g, at_once, stream); break;
    case HASH_POSEIDON2: merkle_launch<HASH_POSEIDON2>(digests, caps, leaves, g, at_once, stream); break;
    case HASH_MONOLITH: merkle_launch<HASH_MONOLITH>(digests, caps, leaves, g, at_once, stream); break;
    default:
        err = "unsupported hash_type " + std::to_string(hash_type);
        return false;
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        err = cudaGetErrorString(e);
        return false;
    }
    return true;
}

cudaError_t oob_take_merkle(uint64_t r[4]) { return oob_take_local(r); }

}  // namespace zk
