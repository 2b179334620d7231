// merkle.cuh -- linear-layout Merkle forest builder (device side).
//
// Replaces native/merkle/merkle.cu:24-280 of zeknox.  Layout (unchanged, it is
// the ABI): 2^cap_height subtrees of L leaves; subtree k owns digests
// [k(2L-2), (k+1)(2L-2)); in it the level with 2^r nodes starts at 2^r - 2,
// node i of a level has children 2(i+1)+start and 2(i+1)+1+start of the level
// below, leaf digests start at L-2, and the subtree root H2(d[0], d[1]) is
// cap[k].
//
// Kernel structure (B200-first instead of one launch per level):
//   * leaf kernel: one thread per leaf runs the sponge with the state in
//     registers (nothing else, so no warp idles on a barrier), or a warp 8, 16
//     or 32 leaves with the linear layers on the tensor cores; rows of up to
//     4 words are copied;
//   * level kernel: one thread per node of one level, for the wide levels
//     just above the leaves (and for levels a tail CTA cannot hold);
//   * fold kernel: each CTA folds T consecutive nodes log2(T) levels up in
//     shared memory, writing every node, and the caps of subtrees that fit;
//   * tail kernel: one CTA per subtree folds the remaining levels in shared
//     memory and writes the cap.
#pragma once
#include <stdint.h>

#include "bounds.cuh"
#include "hash.cuh"
#include "hash_mma.cuh"

namespace zk {

struct MerkleGeom {
    uint64_t n_leaves;
    uint64_t leaf_size;
    uint64_t sub_leaves;   // L
    uint64_t sub_digests;  // 2L - 2
    uint32_t log_sub;      // log2 L
    uint32_t n_caps;
};

__device__ __forceinline__ uint64_t merkle_node_index(const MerkleGeom &g, uint64_t first_leaf, uint32_t level_u)
{
    // node at height level_u (leaves are height 0) covering leaves starting at first_leaf
    uint64_t k = first_leaf >> g.log_sub;
    uint64_t in_sub = first_leaf & (g.sub_leaves - 1);
    uint64_t level_nodes = g.sub_leaves >> level_u;
    return k * g.sub_digests + (level_nodes - 2) + (in_sub >> level_u);
}

// Words of the digest buffer and of the leaves (the extents the checked build
// tests accesses against).
__device__ __forceinline__ uint64_t merkle_digest_words(const MerkleGeom &g) { return 4 * (uint64_t)g.n_caps * g.sub_digests; }
__device__ __forceinline__ uint64_t merkle_leaf_words(const MerkleGeom &g) { return g.n_leaves * g.leaf_size; }

template <int H>
__device__ __forceinline__ void leaf_hash(const uint64_t *__restrict__ row, uint64_t len, uint64_t out[4])
{
    hash_one<H>(row, len, out);
}

// Where leaf i's digest goes: a digest, or with caps == leaves the cap (digests
// untouched).  Null when the checked build finds it or the leaf out of range.
__device__ __forceinline__ uint64_t *merkle_leaf_dst(uint64_t i, uint64_t *digests, uint64_t *caps, const MerkleGeom &g)
{
    if (g.sub_leaves == 1 ? !ZK_IN_BOUNDS(4 * i + 3, 4 * (uint64_t)g.n_caps, OOB_MERKLE_CAP)
                          : !ZK_IN_BOUNDS(4 * merkle_node_index(g, i, 0) + 3, merkle_digest_words(g), OOB_MERKLE_DIGEST))
        return nullptr;
    if (g.leaf_size && !ZK_IN_BOUNDS((i + 1) * g.leaf_size - 1, merkle_leaf_words(g), OOB_MERKLE_LEAF)) return nullptr;
    return g.sub_leaves == 1 ? caps + 4 * i : digests + 4 * merkle_node_index(g, i, 0);
}

// Leaf digests only: one thread per leaf, no shared memory, no barriers, so
// every warp stays on the hash for the whole kernel.
template <int H, int T>
__device__ __forceinline__ void merkle_leaf_body(const uint64_t *__restrict__ leaves, uint64_t *__restrict__ digests,
                                                 uint64_t *__restrict__ caps, const MerkleGeom &g)
{
    const uint64_t i = (uint64_t)blockIdx.x * T + threadIdx.x;
    if (i >= g.n_leaves) return;
    uint64_t *dst = merkle_leaf_dst(i, digests, caps, g);
    if (!dst) return;
    uint64_t d[4];
    if (H == HASH_KECCAK && g.leaf_size < 4) {
        // Keccak copies a < 4-word leaf and leaves the other digest words as
        // they are in the output buffer (native/keccak/keccak.cu:118-121)
#pragma unroll
        for (int q = 0; q < 4; q++) d[q] = dst[q];
    }
    leaf_hash<H>(leaves + i * g.leaf_size, g.leaf_size, d);
#pragma unroll
    for (int q = 0; q < 4; q++) dst[q] = d[q];
}

template <int H, int T>
__global__ void __launch_bounds__(T)
    merkle_leaf_kernel(const uint64_t *__restrict__ leaves, uint64_t *__restrict__ digests, uint64_t *__restrict__ caps,
                       MerkleGeom g)
{
    merkle_leaf_body<H, T>(leaves, digests, caps, g);
}

// Leaves of at most 4 words under Plonky2's sponge: the words themselves, zero padded.
template <int T>
__global__ void __launch_bounds__(T)
    merkle_leaf_copy_kernel(const uint64_t *__restrict__ leaves, uint64_t *__restrict__ digests, uint64_t *__restrict__ caps,
                            MerkleGeom g)
{
    const uint64_t i = (uint64_t)blockIdx.x * T + threadIdx.x;
    if (i >= g.n_leaves) return;
    uint64_t *dst = merkle_leaf_dst(i, digests, caps, g);
    if (!dst) return;
#pragma unroll
    for (uint64_t q = 0; q < 4; q++) dst[q] = q < g.leaf_size ? leaves[i * g.leaf_size + q] : 0;
}

// Folds stored digests upwards from height u0 (0 = leaf digests): each CTA
// takes T consecutive nodes of that height and computes every node above them
// whose subtree lies in the CTA (up to log2 T levels, or up to the subtree's
// two top nodes), writing each node; when whole subtrees fit in the CTA it
// also writes their caps.
template <int H, int T>
__global__ void __launch_bounds__(T) merkle_fold_kernel(uint64_t *__restrict__ digests, uint64_t *__restrict__ caps,
                                                        MerkleGeom g, uint32_t u0)
{
    __shared__ uint64_t node[T][4];
    const uint64_t count = g.n_leaves >> u0;     // nodes at height u0
    const uint64_t i0 = (uint64_t)blockIdx.x * T;  // first node of this CTA (height u0)
    const uint32_t t = threadIdx.x;
    const uint64_t cta_nodes = count - i0 < (uint64_t)T ? count - i0 : (uint64_t)T;
    if (t < cta_nodes) {
        const uint64_t di = merkle_node_index(g, (i0 + t) << u0, u0);
        const bool ok = ZK_IN_BOUNDS(4 * di + 3, merkle_digest_words(g), OOB_MERKLE_NODE);
#pragma unroll
        for (int q = 0; q < 4; q++) node[t][q] = ok ? digests[4 * di + q] : 0;
    }
    const uint32_t top = g.log_sub - 1;  // highest stored height
    uint32_t U = 0;
    while ((1u << (U + 1)) <= T && u0 + U + 1 <= top) U++;
    for (uint32_t v = 1; v <= U; v++) {
        __syncthreads();
        const uint32_t nodes = T >> v;
        uint64_t h[4];
        const bool act = t < nodes && ((uint64_t)t << v) < cta_nodes;
        if (act) {
            hash_two<H>(node[2 * t], node[2 * t + 1], h);
            const uint64_t di = merkle_node_index(g, (i0 + ((uint64_t)t << v)) << u0, u0 + v);
            if (ZK_IN_BOUNDS(4 * di + 3, merkle_digest_words(g), OOB_MERKLE_DIGEST)) {
#pragma unroll
                for (int q = 0; q < 4; q++) digests[4 * di + q] = h[q];
            }
        }
        __syncthreads();
        if (act) {
#pragma unroll
            for (int q = 0; q < 4; q++) node[t][q] = h[q];
        }
    }
    const uint64_t sub_nodes = g.sub_leaves >> u0;  // height-u0 nodes per subtree
    if (u0 + U == top && sub_nodes <= (uint64_t)T) {
        __syncthreads();
        const uint32_t subs = (uint32_t)(cta_nodes / sub_nodes);
        if (t < subs) {
            uint64_t h[4];
            hash_two<H>(node[2 * t], node[2 * t + 1], h);
            const uint64_t k = ((i0 << u0) >> g.log_sub) + t;
            if (ZK_IN_BOUNDS(4 * k + 3, 4 * (uint64_t)g.n_caps, OOB_MERKLE_CAP)) {
#pragma unroll
                for (int q = 0; q < 4; q++) caps[4 * k + q] = h[q];
            }
        }
    }
}

// One CTA per subtree: starting from the stored level of height u0 (m nodes per
// subtree, 2 < m <= MAXM), fold to 2 nodes and write the cap.  Two shared
// buffers (MAXM and MAXM/2 digests) alternate between levels.
template <int H, int MAXM>
__global__ void __launch_bounds__(256) merkle_tail_kernel(uint64_t *__restrict__ digests, uint64_t *__restrict__ caps,
                                                          MerkleGeom g, uint32_t u0)
{
    __shared__ uint64_t bufa[MAXM][4];
    __shared__ uint64_t bufb[MAXM / 2][4];
    const uint64_t k = blockIdx.x;
    uint64_t *sub = digests + k * g.sub_digests * 4;
    const uint64_t sub0 = k * g.sub_digests * 4;  // sub's first word in the digest buffer
    uint32_t m = (uint32_t)(g.sub_leaves >> u0);
    for (uint32_t j = threadIdx.x; j < m; j += blockDim.x) {
        const bool ok = ZK_IN_BOUNDS(sub0 + 4 * (m - 2 + j) + 3, merkle_digest_words(g), OOB_MERKLE_NODE);
#pragma unroll
        for (int q = 0; q < 4; q++) bufa[j][q] = ok ? sub[4 * (m - 2 + j) + q] : 0;
    }
    uint64_t(*src)[4] = bufa;
    uint64_t(*dst)[4] = bufb;
    while (m > 2) {
        __syncthreads();
        uint32_t half = m / 2;
        for (uint32_t j = threadIdx.x; j < half; j += blockDim.x) {
            uint64_t h[4];
            hash_two<H>(src[2 * j], src[2 * j + 1], h);
            const bool ok = ZK_IN_BOUNDS(sub0 + 4 * (half - 2 + j) + 3, merkle_digest_words(g), OOB_MERKLE_DIGEST);
#pragma unroll
            for (int q = 0; q < 4; q++) {
                if (ok) sub[4 * (half - 2 + j) + q] = h[q];
                dst[j][q] = h[q];
            }
        }
        uint64_t(*tmp)[4] = src;
        src = dst;
        dst = tmp;
        m = half;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        uint64_t h[4];
        hash_two<H>(src[0], src[1], h);
        if (ZK_IN_BOUNDS(4 * k + 3, 4 * (uint64_t)g.n_caps, OOB_MERKLE_CAP)) {
#pragma unroll
            for (int q = 0; q < 4; q++) caps[4 * k + q] = h[q];
        }
    }
}

// One level, node-parallel, for very large subtrees (m > tail capacity).
template <int H>
__global__ void merkle_level_kernel(uint64_t *__restrict__ digests, MerkleGeom g, uint32_t u)
{
    uint64_t per_sub = g.sub_leaves >> u;
    uint64_t total = per_sub * g.n_caps;
    for (uint64_t x = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; x < total; x += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t k = x / per_sub, j = x % per_sub;
        uint64_t *sub = digests + k * g.sub_digests * 4;
        uint64_t start = per_sub - 2, child = 2 * per_sub - 2;
        const uint64_t sub0 = k * g.sub_digests * 4;
        if (!ZK_IN_BOUNDS(sub0 + 4 * (child + 2 * j + 1) + 3, merkle_digest_words(g), OOB_MERKLE_NODE) ||
            !ZK_IN_BOUNDS(sub0 + 4 * (start + j) + 3, merkle_digest_words(g), OOB_MERKLE_DIGEST))
            continue;
        uint64_t h[4];
        hash_two<H>(sub + 4 * (child + 2 * j), sub + 4 * (child + 2 * j + 1), h);
#pragma unroll
        for (int q = 0; q < 4; q++) sub[4 * (start + j) + q] = h[q];
    }
}

// ------------------------------------------------------ tensor-core kernels
//
// Poseidon and Poseidon2 with the linear layers on the tensor cores
// (hash_mma.cuh): a warp hashes 8 * NS leaves or nodes, row q * 8 + g of its
// span being state q of quad g.  Rows past the end repeat the last one and
// store nothing.

// Threads per SM the register budget of the 32-state form aims at: 640 (96
// registers) where the GPU is full (Poseidon2 2^20 x 135: 14.23 ms against
// 14.32 at 512; 768 and 1024 spill: 15.2 and 19.8 against 14.9 in an earlier
// form), 512 (128 registers) for the one-warp CTAs of forests that give an SM a
// handful of warps, whose S-boxes then overlap further (2^15 x 135: 763
// against 863 us).
__host__ __device__ constexpr int mma_threads_per_sm(int t) { return t == 32 ? 512 : 640; }

// Leaf digests (leaf_size > 4: shorter leaves are copied, not hashed).
template <int H, int NS, int T>
__global__ void __launch_bounds__(T, NS == 4 ? mma_threads_per_sm(T) / T : 1)
    merkle_leaf_mma_kernel(const uint64_t *__restrict__ leaves, uint64_t *__restrict__ digests,
                           uint64_t *__restrict__ caps, MerkleGeom g)
{
    __shared__ __align__(16) uint32_t sm[T / 32][MmaSmem<NS>::template words<H>()];
    const uint32_t warp = threadIdx.x >> 5, quad = (threadIdx.x & 31) >> 2, t = threadIdx.x & 3;
    const uint64_t first = ((uint64_t)blockIdx.x * (T / 32) + warp) * (8 * NS) + quad;
    if (first - quad >= g.n_leaves) return;  // the whole warp is past the end
    uint64_t d[NS];
    auto row = [&](int q) {
        const uint64_t i = first + 8 * q < g.n_leaves ? first + 8 * q : g.n_leaves - 1;
        return leaves + (ZK_IN_BOUNDS((i + 1) * g.leaf_size - 1, merkle_leaf_words(g), OOB_MERKLE_LEAF) ? i : 0) * g.leaf_size;
    };
    sponge_hash_mma<H, NS>(row, g.leaf_size, sm[warp], d);
#pragma unroll
    for (int q = 0; q < NS; q++) {
        const uint64_t i = first + 8 * q;
        if (i >= g.n_leaves) continue;
        // caps == leaves: the leaf hashes are the caps
        if (g.sub_leaves == 1) {
            if (ZK_IN_BOUNDS(4 * i + t, 4 * (uint64_t)g.n_caps, OOB_MERKLE_CAP)) caps[4 * i + t] = d[q];
        } else {
            const uint64_t w = 4 * merkle_node_index(g, i, 0) + t;
            if (ZK_IN_BOUNDS(w, merkle_digest_words(g), OOB_MERKLE_DIGEST)) digests[w] = d[q];
        }
    }
}

// One level of height u, every node of every subtree.
template <int H, int NS, int T>
__global__ void __launch_bounds__(T, NS == 4 ? mma_threads_per_sm(T) / T : 1)
    merkle_level_mma_kernel(uint64_t *__restrict__ digests, MerkleGeom g, uint32_t u)
{
    __shared__ __align__(16) uint32_t sm[T / 32][MmaSmem<NS>::template words<H>()];
    const uint32_t warp = threadIdx.x >> 5, quad = (threadIdx.x & 31) >> 2, t = threadIdx.x & 3;
    const uint64_t total = g.n_leaves >> u;
    const uint64_t first = ((uint64_t)blockIdx.x * (T / 32) + warp) * (8 * NS) + quad;
    if (first - quad >= total) return;
    uint64_t d[NS];
    auto row = [&](int q) {
        const uint64_t x = first + 8 * q < total ? first + 8 * q : total - 1;
        // the two children of a node are neighbours: eight consecutive words
        const uint64_t w = 4 * merkle_node_index(g, x << u, u - 1);
        return (const uint64_t *)digests + (ZK_IN_BOUNDS(w + 7, merkle_digest_words(g), OOB_MERKLE_NODE) ? w : 0);
    };
    sponge_hash_mma<H, NS>(row, 8, sm[warp], d);
#pragma unroll
    for (int q = 0; q < NS; q++) {
        const uint64_t x = first + 8 * q;
        if (x >= total) continue;
        const uint64_t w = 4 * merkle_node_index(g, x << u, u) + t;
        if (ZK_IN_BOUNDS(w, merkle_digest_words(g), OOB_MERKLE_DIGEST)) digests[w] = d[q];
    }
}

// merkle_fold_kernel for the tensor-core hashes: a CTA of four warps takes
// MMA_FOLD_IN consecutive nodes of height u0 (its first level is one
// permutation per quad of threads) and computes every node above them whose
// subtree lies in the CTA, and the caps of subtrees that fit.  What these
// narrow levels wait on is the latency of one permutation per level: 8 states
// per warp (NS = 1), a third of the lanes' S-boxes per thread.  TSM: the tables
// are copied to dynamic shared memory first, when a CTA has an SM to itself.
// L1 starts empty at every launch, and a warp alone fetches the tables' lines
// one after another on its first permutation.
static constexpr uint32_t MMA_FOLD_IN = 64;

template <int H, bool TSM>
__global__ void __launch_bounds__(128) merkle_fold_mma_kernel(uint64_t *__restrict__ digests, uint64_t *__restrict__ caps,
                                                              MerkleGeom g, uint32_t u0)
{
    extern __shared__ __align__(16) uint32_t table_copy[];
    __shared__ __align__(16) uint32_t sm[4][MmaSmem<1>::words<H>()];
    __shared__ uint64_t node[MMA_FOLD_IN][4];
    if constexpr (TSM) {
        const uint4 *table = (const uint4 *)mma_table<H>();
#pragma unroll 12
        for (uint32_t k = threadIdx.x; k < mma_table_words<H>() / 4; k += 128)
            ((uint4 *)table_copy)[k] = __ldg(table + k);
    }
    const uint32_t quad = threadIdx.x >> 2, t = threadIdx.x & 3, warp = threadIdx.x >> 5;
    const uint32_t wq = quad & ~7u;  // first quad of this warp
    const uint64_t count = g.n_leaves >> u0;
    const uint64_t i0 = (uint64_t)blockIdx.x * MMA_FOLD_IN;
    const uint64_t cta_nodes = count - i0 < MMA_FOLD_IN ? count - i0 : MMA_FOLD_IN;
    for (uint32_t k = threadIdx.x; k < 4 * cta_nodes; k += 128) {
        const uint64_t wi = 4 * merkle_node_index(g, (i0 + (k >> 2)) << u0, u0) + (k & 3);
        node[k >> 2][k & 3] = ZK_IN_BOUNDS(wi, merkle_digest_words(g), OOB_MERKLE_NODE) ? digests[wi] : 0;
    }
    const uint32_t top = g.log_sub - 1;
    uint32_t U = 0;
    while ((1u << (U + 1)) <= MMA_FOLD_IN && u0 + U + 1 <= top) U++;
    const uint64_t sub_nodes = g.sub_leaves >> u0;
    // levels 1..U, then the caps when whole subtrees fit in the CTA
    const uint32_t last = u0 + U == top && sub_nodes <= MMA_FOLD_IN ? U + 1 : U;
#pragma unroll 1
    for (uint32_t v = 1; v <= last; v++) {
        __syncthreads();
        // nodes of this level in the CTA (at the caps: its subtrees)
        const uint32_t nodes = v <= U ? (uint32_t)((cta_nodes + (1u << v) - 1) >> v) : (uint32_t)(cta_nodes / sub_nodes);
        const bool act = quad < nodes;
        uint64_t h[1];
        if (wq < nodes) {
            // a quad with no node repeats its warp's first
            const uint64_t *src = &node[2 * (act ? quad : wq)][0];
            if constexpr (TSM) sponge_hash_mma<H, 1, true>([&](int) { return src; }, 8, sm[warp], h, table_copy);
            else sponge_hash_mma<H, 1>([&](int) { return src; }, 8, sm[warp], h);
            if (act && v <= U) {
                const uint64_t w = 4 * merkle_node_index(g, (i0 + ((uint64_t)quad << v)) << u0, u0 + v) + t;
                if (ZK_IN_BOUNDS(w, merkle_digest_words(g), OOB_MERKLE_DIGEST)) digests[w] = h[0];
            } else if (act) {
                const uint64_t w = 4 * (((i0 << u0) >> g.log_sub) + quad) + t;
                if (ZK_IN_BOUNDS(w, 4 * (uint64_t)g.n_caps, OOB_MERKLE_CAP)) caps[w] = h[0];
            }
        }
        __syncthreads();
        if (act && v <= U) node[quad][t] = h[0];
    }
}

#if ZK_BN128_LIMBS29
// ---------------------------------------------- Poseidon-BN128, five threads a state
//
// (bn254_29.cuh.)  Groups without a leaf or node repeat their warp's last one
// and store nothing.

// Leaf digests (leaf_size > 4), six per warp.
template <int T>
__global__ void __launch_bounds__(T)
    merkle_leaf_bn128_kernel(const uint64_t *__restrict__ leaves, uint64_t *__restrict__ digests,
                             uint64_t *__restrict__ caps, MerkleGeom g)
{
    Fr29Group grp;
    grp.init();
    const uint64_t first = ((uint64_t)blockIdx.x * (T / 32) + (threadIdx.x >> 5)) * 6;
    if (first >= g.n_leaves) return;  // the whole warp is past the end
    const uint64_t i = first + grp.base / 5;
    const bool act = grp.live && i < g.n_leaves;
    const uint64_t row = act ? i : first;
    const bool ok = ZK_IN_BOUNDS((row + 1) * g.leaf_size - 1, merkle_leaf_words(g), OOB_MERKLE_LEAF);
    uint64_t d[3];
    sponge_bn128_group(leaves + (ok ? row : 0) * g.leaf_size, g.leaf_size, d, grp);
    if (!act || !ok || grp.i == 0 || grp.i > 2) return;
#pragma unroll
    for (uint32_t q = 0; q < 3; q++) {
        const uint64_t w = 3 * (grp.i - 1) + q;  // digest word
        if (w > 3) continue;
        if (g.sub_leaves == 1) {
            if (ZK_IN_BOUNDS(4 * i + w, 4 * (uint64_t)g.n_caps, OOB_MERKLE_CAP)) caps[4 * i + w] = d[q];
        } else {
            const uint64_t at = 4 * merkle_node_index(g, i, 0) + w;
            if (ZK_IN_BOUNDS(at, merkle_digest_words(g), OOB_MERKLE_DIGEST)) digests[at] = d[q];
        }
    }
}

// merkle_fold_mma_kernel with five threads a state: six warps, 36 groups for
// the 32 nodes of a CTA's first level.
static __global__ void __launch_bounds__(192)
    merkle_fold_bn128_kernel(uint64_t *__restrict__ digests, uint64_t *__restrict__ caps, MerkleGeom g, uint32_t u0)
{
    __shared__ uint64_t node[MMA_FOLD_IN][4];
    Fr29Group grp;
    grp.init();
    const uint32_t wf = (threadIdx.x >> 5) * 6, quint = wf + grp.base / 5;  // first group of the warp, this group
    const uint64_t count = g.n_leaves >> u0;
    const uint64_t i0 = (uint64_t)blockIdx.x * MMA_FOLD_IN;
    const uint64_t cta_nodes = count - i0 < MMA_FOLD_IN ? count - i0 : MMA_FOLD_IN;
    for (uint32_t k = threadIdx.x; k < 4 * cta_nodes; k += 192) {
        const uint64_t wi = 4 * merkle_node_index(g, (i0 + (k >> 2)) << u0, u0) + (k & 3);
        node[k >> 2][k & 3] = ZK_IN_BOUNDS(wi, merkle_digest_words(g), OOB_MERKLE_NODE) ? digests[wi] : 0;
    }
    const uint32_t top = g.log_sub - 1;
    uint32_t U = 0;
    while ((1u << (U + 1)) <= MMA_FOLD_IN && u0 + U + 1 <= top) U++;
    const uint64_t sub_nodes = g.sub_leaves >> u0;
    const uint32_t last = u0 + U == top && sub_nodes <= MMA_FOLD_IN ? U + 1 : U;
#pragma unroll 1
    for (uint32_t v = 1; v <= last; v++) {
        __syncthreads();
        const uint32_t nodes = v <= U ? (uint32_t)((cta_nodes + (1u << v) - 1) >> v) : (uint32_t)(cta_nodes / sub_nodes);
        const bool act = grp.live && quint < nodes;
        uint64_t h[3];
        if (wf < nodes) {
            sponge_bn128_group(&node[2 * (act ? quint : wf)][0], 8, h, grp);
            if (act && (grp.i == 1 || grp.i == 2)) {
#pragma unroll
                for (uint32_t q = 0; q < 3; q++) {
                    const uint32_t w = 3 * (grp.i - 1) + q;
                    if (w > 3) continue;
                    if (v <= U) {
                        const uint64_t at = 4 * merkle_node_index(g, (i0 + ((uint64_t)quint << v)) << u0, u0 + v) + w;
                        if (ZK_IN_BOUNDS(at, merkle_digest_words(g), OOB_MERKLE_DIGEST)) digests[at] = h[q];
                    } else {
                        const uint64_t at = 4 * (((i0 << u0) >> g.log_sub) + quint) + w;
                        if (ZK_IN_BOUNDS(at, 4 * (uint64_t)g.n_caps, OOB_MERKLE_CAP)) caps[at] = h[q];
                    }
                }
            }
        }
        __syncthreads();
        if (act && v <= U && (grp.i == 1 || grp.i == 2)) {
#pragma unroll
            for (uint32_t q = 0; q < 3; q++) {
                const uint32_t w = 3 * (grp.i - 1) + q;
                if (w <= 3) node[quint][w] = h[q];
            }
        }
    }
}
#endif  // ZK_BN128_LIMBS29

}  // namespace zk
